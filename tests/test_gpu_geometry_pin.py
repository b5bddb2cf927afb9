"""The CUDA geometry routines checked directly, without a transport run in
between: howfar (region entered, step, state after the call) and hownear of
the phantom, the DYNVMLC and the secondary jaws, run on the device by
gegs_probe_geometry on given particle states.

* against the reference's own routines: the outputs the reference harness
  recorded for 9 559 states of the full CT head 5-field geometry
  (tests/golden/ref_pin_c3.npz, written by tests/golden/make_ref_fixtures.py);
* against the oracle: every particle state that enters the photon and
  electron stages of oracle runs of the full C1, C2 and C3 geometries, at the
  transport's step and at short steps.

Bit for bit."""
import pathlib

import numpy as np
import pytest

import refpin_cases as RC

GOLDEN = pathlib.Path(__file__).resolve().parent / "golden"


def _engine(engine, job):
    sh = job.scene()
    engine.set_physics(job.physics)
    engine.set_scene(sh)
    return sh


def _compare(res, region, t, particle, tperp):
    assert np.array_equal(res["region"], region), "howfar region"
    assert res["t"].tobytes() == np.asarray(t, np.float32).tobytes(), "howfar step"
    assert res["tperp"].tobytes() == np.asarray(tperp, np.float32).tobytes(), "hownear distance"
    assert res["particle"].tobytes() == np.ascontiguousarray(particle).tobytes(), "state after howfar"


@pytest.mark.gpu
def test_device_geometry_equals_the_reference_recordings(engine):
    z = np.load(GOLDEN / "ref_pin_c3.npz")
    _engine(engine, RC.job("c3"))
    res = engine.probe_geometry(z["geom_in"], z["geom_t_in"])
    assert len(res["region"]) == len(z["geom_in"]) > 9000
    assert set(np.unique(z["geom_in"]["module"])) >= {1, 2, 3, 6}       # jaws Y, jaws X, MLC, phantom
    _compare(res, z["geom_region"], z["geom_t"], z["geom_out"], z["geom_tperp"])


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c1", "c2", "c3"])
def test_device_geometry_equals_the_oracle(engine, name):
    from oracle import refpin as R
    job = RC.job(name)
    sh = _engine(engine, job)
    pair = R.OraclePair(job.physics, sh)
    cap = pair.capture(0, job.histories, every=1, cap_n=60000)
    parts = np.concatenate([cap[0], cap[5]])                         # photon and electron stage entries
    assert len(parts) > 5000
    rng = np.random.default_rng(11)
    for t_in in (np.full(len(parts), 1e3, np.float32), rng.exponential(0.3, len(parts)).astype(np.float32)):
        want = pair.geom(parts, t_in)
        res = engine.probe_geometry(parts, t_in)
        _compare(res, want["region"], want["t"], want["particle"], want["tperp"])


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0.0, 1e-6, 1e-4, 2e-3])
def test_device_geometry_at_polygon_vertices_and_edges(engine, offset):
    """Where the polygon routines pick out the edges that they divide for:
    points on, and `offset` cm around, the vertices and edge midpoints of the
    leaf cross sections, the leaf-end outlines and the jaws, with directions
    along the axes (edges parallel to the ray) and oblique ones, in a leaf, in a
    gap, outside, and with the bank known or not. Bit for bit as the oracle."""
    from oracle import refpin as R
    job = RC.job("c3")
    sh = _engine(engine, job)
    pair = R.OraclePair(job.physics, sh)
    cap = pair.capture(0, 2000, every=1, cap_n=20000)
    base = np.concatenate([cap[0], cap[5]])
    rng = np.random.default_rng(29)
    cross = np.ctypeslib.as_array(sh.scene.crossXZ).reshape(60, 16, 2)[:, :14]
    out = []
    for module, n in ((3, 6000), (1, 2000), (2, 2000)):
        have = base[base["module"] == module]
        p = have[rng.integers(0, len(have), n)].copy()
        f = p["field"] = rng.integers(0, len(job.fields), n)
        k = rng.integers(0, 60, n)
        if module == 3:
            leaf = k.astype(np.int8)
            end = np.stack([np.ctypeslib.as_array(sh.scene.fields[i].endnode) for i in range(len(job.fields))])
            a, b = cross[k, k % 14], cross[k, (k + 1) % 14]
            mid = rng.integers(0, 2, n)[:, None] / 2.0
            xz = a + (b - a) * mid
            yz = end[f, k, rng.integers(0, 34, n)]
            on_x = rng.integers(0, 2, n) == 0
            p["x"] = np.where(on_x, xz[:, 0], cross[k].mean(1)[:, 0])
            p["y"] = np.where(on_x, rng.uniform(-8, 8, n), yz[:, 0])
            p["z"] = np.where(on_x, xz[:, 1], yz[:, 1])
            p["leafIndex"] = np.choose(rng.integers(0, 4, n), [leaf, leaf, -np.maximum(leaf, 1), -99])
            p["bank"] = np.choose(rng.integers(0, 4, n), [-1, 0, 1, 2])
            p["region"] = np.where(p["bank"] > 0, 3, 1)
        else:
            geo = "jawsGeomX" if module == 2 else "jawsGeomY"
            v = np.stack([np.ctypeslib.as_array(getattr(sh.scene.fields[i], geo)) for i in range(len(job.fields))])
            q = v[f, rng.integers(0, 8, n)]
            p["y" if module == 2 else "x"] = q[:, 0]
            p["x" if module == 2 else "y"] = rng.uniform(-4, 4, n)
            p["z"] = q[:, 1]
            p["region"] = rng.integers(1, 3, n)
        for c in ("x", "y", "z"):
            p[c] = (p[c] + offset * rng.integers(-1, 2, n)).astype(np.float32)
        d = rng.normal(size=(n, 3)).astype(np.float32)
        d[np.arange(n), rng.integers(0, 3, n)] *= rng.integers(0, 2, n)
        d[np.arange(n), rng.integers(0, 3, n)] *= rng.integers(0, 2, n)
        d[(d == 0).all(1)] = (0, 0, 1)
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        p["u"], p["v"], p["w"] = d[:, 0], d[:, 1], d[:, 2]
        out.append(p)
    parts = np.concatenate(out)
    for t_in in (np.full(len(parts), 1e3, np.float32), rng.exponential(0.3, len(parts)).astype(np.float32)):
        want = pair.geom(parts, t_in)
        res = engine.probe_geometry(parts, t_in)
        _compare(res, want["region"], want["t"], want["particle"], want["tperp"])
