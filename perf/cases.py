"""The calls whose speed counts, over the sizes they are made with.

Transport plans of the package's three geometries (a water cube, a slab under a
point source, a CT head behind jaws and MLC), from a quick look of some ten
thousand histories to a plan's full run; the beamlet gradient; several plans in
one launch; a series of batches for the uncertainty; and what follows a dose:
gamma, interpolation, and the HU ramp that precedes it. Plans of more than a
million histories per field use each phase-space record several times.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gegs_b200 import geometry as G
from gegs_b200 import workloads as W
from gegs_b200.batch import PlanBatch
from gegs_b200.differentiable import BeamletModel, beamlet_dose, objective
from gegs_b200.engine import Engine
from gegs_b200.postprocess import ct_ramp, gamma3d, interp_dose

RECORDS = 1_000_000          # phase-space records of a plan, at most
RAMP_MEDIA = ["AIR700ICRU", "LUNG700ICRU", "ICRUTISSUE700ICRU", "ICRPBONE700ICRU"]


def listed():
    return [
        # a look at a plan while it is set up: few histories, so launches and waves count
        dict(name="water-1e4", kind="plan", scene="water", nx=60, ny=60, nz=60, fields=1, histories=10_000),
        # the water cube at its stated size and count
        dict(name="water-1e6", kind="plan", scene="water", nx=60, ny=60, nz=60, fields=1, histories=1_000_000),
        # the slab at its stated size, read out as dose
        dict(name="slab-5e6", kind="dose", scene="slab", nx=120, ny=120, nz=120, fields=1, histories=5_000_000),
        # the CT head plan with the history count of one optimisation step, where a run's tail counts
        dict(name="head-1e6", kind="plan", scene="head", nx=256, ny=256, nz=120, fields=5, histories=1_000_000),
        # the CT head plan run for a dose
        dict(name="head-16e6", kind="plan", scene="head", nx=256, ny=256, nz=120, fields=5, histories=16_000_000),
        # a CT of another size with other fields: odd dimensions, a history count that nothing divides
        dict(name="head-odd", kind="plan", scene="head", nx=161, ny=117, nz=87, fields=3, histories=3_000_017),
        # one step of the beamlet optimisation: forward dose, objective, gradient by replay
        dict(name="beamlets", kind="beamlets", nx=128, ny=128, nz=96, fields=5, beamlets=20, histories=1_000_000),
        # small plans of several sizes served in one launch
        dict(name="plans", kind="plans", plans=6, size=64, histories=300_000),
        # a run in ten batches for the uncertainty per voxel
        dict(name="uncertainty", kind="uncertainty", scene="slab", nx=120, ny=120, nz=120, fields=1, batches=10,
             histories=2_000_000),
        # two doses of a head compared at 1 % / 1 mm
        dict(name="gamma", kind="gamma", nx=256, ny=256, nz=120),
        # a dose brought to another grid
        dict(name="interp", kind="interp", nx=256, ny=256, nz=120, mx=200, my=200, mz=150),
        # a CT volume turned into media and densities
        dict(name="ct-ramp", kind="ramp", nx=256, ny=256, nz=120),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["plan", "plan", "plan", "dose", "beamlets", "plans", "uncertainty", "gamma", "interp", "ramp"])
    dims = dict(nx=log(64, 256), ny=log(64, 256), nz=log(64, 120))
    if kind in ("gamma", "ramp"):
        return dict(kind=kind, **dims)
    if kind == "interp":
        return dict(kind=kind, **dims, mx=log(40, 256), my=log(40, 256), mz=log(40, 160))
    if kind == "plans":
        return dict(kind=kind, plans=rng.randint(2, 6), size=log(48, 96), histories=log(100_000, 600_000))
    if kind == "beamlets":
        return dict(kind=kind, nx=log(64, 160), ny=log(64, 160), nz=log(48, 96), fields=rng.randint(1, 7),
                    beamlets=rng.randint(8, 20), histories=log(100_000, 2_000_000))
    scene = rng.choice(["water", "slab", "head", "head"])
    histories = log(10_000, 8_000_000)
    if scene != "head":
        n = log(48, 128)
        dims = dict(nx=n, ny=n, nz=n)
    case = dict(kind=kind, scene=scene, **dims, fields=rng.randint(1, 7) if scene == "head" else 1, histories=histories)
    if kind == "uncertainty":
        case["batches"] = rng.randint(4, 12)
        case["histories"] = max(histories, 100_000)
    return case


# ---- inputs ------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _plan_of(scene, nx, ny, nz):
    """The parts of a plan that a user's program has once: tables, phantom, beam line."""
    if scene == "water":
        return W.config1(histories=1, n=nx, voxel=30.0 / nx)
    if scene == "slab":
        return W.config2(histories=1, nphsp=1, n=nx)
    return W.config3(histories=1, nphsp=1, dims=(nx, ny, nz), angles=(0.0,))


def _job(scene, nx, ny, nz, fields, histories, seed):
    """A plan of the scene with its phase space, fields and leaf positions drawn from the seed."""
    base = _plan_of(scene, nx, ny, nz)
    rng = np.random.default_rng(seed)
    n = min(histories, RECORDS)
    beam = dict(base.beam)
    if scene == "water":
        rec = np.zeros(n, base.phsp.dtype)
        rec["e"], rec["wt"] = 1.25, 1.0
        rec["x"], rec["y"] = rng.uniform(-5, 5, n), rng.uniform(-5, 5, n)
        c, s = G.gantry_cos_sin(0.0)
        fs = [dict(cos_angle=c, sin_angle=s, hist_begin=0, hist_end=histories, nrepeat=(histories - 1) // n)]
    elif scene == "slab":
        rec = W.point_source_phsp(rng, n, z_phsp=beam["z_phsp"], half_x=5.0, half_y=5.0)
        c, s = G.gantry_cos_sin(0.0)
        fs = [dict(cos_angle=c, sin_angle=s, hist_begin=0, hist_end=histories, nrepeat=(histories - 1) // n)]
    else:
        rec = W.point_source_phsp(rng, n, z_phsp=beam["z_phsp"], half_x=7.0, half_y=7.0)
        mlc, jaws, fs, per = base.meta["mlc"], base.meta["jaws"], [], histories // fields
        for i, a in enumerate(np.linspace(0.0, 360.0, fields, endpoint=False)):
            c, s = G.gantry_cos_sin(float(a))
            pos = W.mlc_tips(rng, half=6.0)
            f = dict(cos_angle=c, sin_angle=s, hist_begin=i * per,
                     hist_end=(i + 1) * per if i < fields - 1 else histories, nrepeat=max(0, (per - 1) // n))
            f.update(G.secjaws_polygons(jaws, -6.0, 6.0, -6.0, 6.0, 100.0))
            f["endnode"] = G.leaf_endnodes(beam["mlc"]["crossYZ"], pos, mlc.zmin, mlc.zthick, 100.0)
            fs.append(f)
    return W.Job(base.name, base.media, base.physics, base.phantom, beam, fs, rec, histories, meta=dict(seed=seed + 1))


def _engine(job):
    e = Engine(0)
    e.set_physics(job.physics)
    e.set_scene(job.scene())
    return e


def _pinned(n):
    return torch.empty(n, dtype=torch.int64, pin_memory=True).numpy()


@functools.lru_cache(maxsize=4)
def _volumes(nx, ny, nz):
    """Target and organ of the head, as masks over its voxels."""
    job = _plan_of("head", nx, ny, nz)
    return (W.ellipsoid_mask(job, (0.0, 0.0, 0.0), (2.5, 2.0, 3.0)), W.ellipsoid_mask(job, (1.5, 0.5, 0.0), (1.0, 1.5, 2.0)))


def _dose_grid(rng, nx, ny, nz):
    """A dose as two crossing beams leave it: a high region, its edges, and little elsewhere."""
    x, y, z = (np.linspace(-1, 1, n, dtype=np.float32) for n in (nx, ny, nz))
    edge = lambda v, w: 1.0 / (1.0 + np.exp((np.abs(v) - w) * 30.0))
    c = rng.uniform(-0.1, 0.1, 3).astype(np.float32)
    a = (edge(z - c[2], 0.45)[:, None, None] * np.exp(-0.5 * (y + 1))[None, :, None] * edge(x - c[0], 0.4)[None, None, :])
    b = (edge(z - c[2], 0.45)[:, None, None] * edge(y - c[1], 0.4)[None, :, None] * np.exp(-0.5 * (x + 1))[None, None, :])
    return (a + b + 0.01).astype(np.float32)


def _noise(rng, shape, sigma):
    return (1.0 + np.float32(sigma) * rng.standard_normal(shape, dtype=np.float32)).astype(np.float32)


def _bounds(n, size):
    return (np.arange(n + 1, dtype=np.float64) * size - n * size / 2).astype(np.float32)


def _output_grid(case):
    """Start, spacing and dims of the interpolated grid: inside the phantom, with a rim outside its voxel centres."""
    size = (case["nx"] * 0.1, case["ny"] * 0.1, case["nz"] * 0.25)
    dims = (case["mx"], case["my"], case["mz"])
    step = tuple(s * 1.01 / m for s, m in zip(size, dims))
    return tuple(-0.503 * s for s in size), step, dims


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("plan", "dose", "uncertainty"):
        job = _job(case["scene"], case["nx"], case["ny"], case["nz"], case["fields"], case["histories"], seed)
        e = _engine(job)
        return dict(kind=kind, engine=e, histories=case["histories"], out=_pinned(e.nvox) if kind == "plan" else None,
                    mass=job.voxel_mass() if kind == "dose" else None, batches=case.get("batches"))
    if kind == "beamlets":
        job = _job("head", case["nx"], case["ny"], case["nz"], case["fields"], case["histories"], seed)
        nb = case["beamlets"]
        w = (1.0 + rng.uniform(0.0, 0.2, case["fields"] * nb * nb)).astype(np.float32)
        job.beam["beamlets"] = dict(nx=nb, ny=nb, x0=-5.0, y0=-5.0, dx=10.0 / nb, dy=10.0 / nb, weights=w)
        target, organ = _volumes(case["nx"], case["ny"], case["nz"])
        model = BeamletModel(_engine(job), job)
        model.calibrate(w, target, 50.0)
        return dict(kind=kind, model=model, w=torch.tensor(w.astype(np.float64), requires_grad=True), target=target,
                    organ=organ)
    if kind == "plans":
        jobs = []
        for k in range(case["plans"]):
            n, h = case["size"] + 11 * k, case["histories"] * (k + 2) // 3
            if k % 2 == 0:
                jobs.append(_job("slab", n, n, n, 1, h, seed * 16 + k))
            else:
                jobs.append(_job("head", n, n + 5, n - 3, 1 + (2 * k) % 7, h, seed * 16 + k))
        return dict(kind=kind, batch=PlanBatch(jobs))
    shape = (case["nz"], case["ny"], case["nx"])
    if kind == "gamma":
        ref = _dose_grid(rng, case["nx"], case["ny"], case["nz"])
        ev = np.roll(ref, 1, axis=2) * _noise(rng, shape, 0.01)
        return dict(kind=kind, ref=ref * _noise(rng, shape, 0.005), ev=ev, spacing=(0.1, 0.1, 0.25))
    if kind == "interp":
        dose = _dose_grid(rng, case["nx"], case["ny"], case["nz"]) * _noise(rng, shape, 0.01)
        b = [_bounds(case["nx"], 0.1), _bounds(case["ny"], 0.1), _bounds(case["nz"], 0.25)]
        return dict(kind=kind, dose=dose, bounds=b, grid=_output_grid(case))
    hu = _plan_of("head", case["nx"], case["ny"], case["nz"]).phantom["hu"].reshape(-1)
    hu = hu + rng.integers(-20, 21, hu.size, dtype=np.int16)
    seg = [(RAMP_MEDIA.index(n), ub, lo, hi) for n, ub, lo, hi in W.CT_RAMP]
    return dict(kind="ramp", hu=hu, segments=seg)


def run(state):
    kind = state["kind"]
    if kind == "plan":
        e = state["engine"]
        e.reset_tally()
        e.run(0, state["histories"])
        return e.tally(out=state["out"])
    if kind == "dose":
        e = state["engine"]
        e.reset_tally()
        e.run(0, state["histories"])
        return e.dose(state["mass"])
    if kind == "uncertainty":
        e, n, h = state["engine"], state["batches"], state["histories"]
        e.stat_begin()
        for b in range(n):
            e.run(b * h // n, (b + 1) * h // n)
            e.stat_fold()
        mean, rel, _ = e.stat_get()
        return mean, rel
    if kind == "beamlets":
        w = state["w"]
        w.grad = None
        dose = beamlet_dose(w, state["model"])
        loss = objective(dose, state["target"], state["organ"])
        loss.backward()
        return dict(dose=dose.detach(), loss=loss.detach(), gradient=w.grad)
    if kind == "plans":
        state["batch"].run()
        return state["batch"].tallies()
    if kind == "gamma":
        return gamma3d(state["ref"], state["ev"], state["spacing"])
    if kind == "interp":
        return interp_dose(state["dose"], *state["bounds"], *state["grid"])
    return ct_ramp(state["hu"], state["segments"], W.CT_LOWER)


# photon and electron steps of a history, and operations of a step: a photon's free path, the distance to its voxel's
# walls and its move; an electron's step length, energy loss, scattering angle and move
STEPS = {"water": (94, 54), "slab": (171, 69), "head": (176, 48)}
PHOTON_STEP, ELECTRON_STEP = 60, 300


def _transport(scene, voxels, histories):
    p, e = STEPS[scene]
    return dict(bytes=28.0 * min(histories, RECORDS) + 16.0 * voxels,
                flops=float(histories) * (p * PHOTON_STEP + e * ELECTRON_STEP))


def work(case):
    """Phase space and regions read once, the tally written once; the steps of a history. A grid read and written once."""
    kind = case["kind"]
    if kind == "plans":
        total = dict(bytes=0.0, flops=0.0)
        for k in range(case["plans"]):
            n, h = case["size"] + 11 * k, case["histories"] * (k + 2) // 3
            one = _transport("head" if k % 2 else "slab", n * (n + 5) * (n - 3) if k % 2 else n ** 3, h)
            total = {q: total[q] + one[q] for q in total}
        return total
    voxels = case["nx"] * case["ny"] * case["nz"]
    if kind in ("plan", "dose", "uncertainty"):
        one = _transport(case["scene"], voxels, case["histories"])
        if kind == "dose":
            one["bytes"] += 12.0 * voxels
        if kind == "uncertainty":
            one["bytes"] += 16.0 * voxels + 40.0 * voxels * case["batches"]
        return one
    if kind == "beamlets":
        one = _transport("head", voxels, case["histories"])
        return dict(bytes=2 * one["bytes"] + 24.0 * voxels, flops=2 * one["flops"])
    if kind == "gamma":
        return dict(bytes=12.0 * voxels, flops=20.0 * voxels)
    if kind == "interp":
        out = case["mx"] * case["my"] * case["mz"]
        return dict(bytes=4.0 * voxels + 4.0 * out, flops=30.0 * out)
    return dict(bytes=8.0 * voxels, flops=6.0 * voxels)


def tolerance(case):
    """Tallies are whole numbers; what is computed from them in 64 bits, and the float grids, by their types."""
    kind = case["kind"]
    if kind in ("plan", "plans"):
        return "exact"
    if kind == "dose":
        return dict(rel=1e-14, max=1e-13)
    if kind == "beamlets":
        return dict(rel=1e-11, max=1e-9)             # the gradient's sums, in any order
    if kind == "uncertainty":
        return dict(rel=1e-9, max=1e-6)              # a difference of sums of squares
    if kind == "gamma":
        return dict(rel=1e-6, max=1e-4)
    if kind == "interp":
        return dict(rel=1e-6, max=1e-4)
    return dict(rel=1e-7, max=1e-6, differ=0.0)


def exact(case, seed):
    """The float grids in 64 bits (a transport has no such values)."""
    kind = case["kind"]
    if kind not in ("gamma", "interp", "ramp"):
        return None
    s = prepare(case, seed)
    if kind == "ramp":
        hu = torch.from_numpy(s["hu"]).double()
        med = torch.full(hu.shape, W.VACUUM_MED, dtype=torch.int32)
        dens = torch.zeros_like(hu)
        lower, todo = float(W.CT_LOWER), hu >= W.CT_LOWER
        for m, ub, lo, hi in s["segments"]:
            sel = todo & (hu <= ub)
            med[sel] = m
            dens[sel] = lo + (hu[sel] - lower) * (hi - lo) / (ub - lower)
            todo &= ~sel
            lower = ub
        med[todo] = s["segments"][-1][0]
        dens[todo] = s["segments"][-1][3]
        return med.numpy().astype(np.uint16), dens.numpy()
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "interp":
        start, step, dims = s["grid"]
        v = torch.from_numpy(s["dose"]).to(dev).double()
        for axis in range(3):                        # x, y, z of the (nz, ny, nx) grid
            b = s["bounds"][axis]
            c = torch.from_numpy(((b[:-1] + b[1:]) / 2)).to(dev).double()
            p = float(np.float32(start[axis])) + float(np.float32(step[axis])) * torch.arange(dims[axis], device=dev, dtype=torch.float64)
            inside = (p > c[0]) & (p < c[-1])
            k = (torch.searchsorted(c, p, right=False) - 1).clamp(0, len(c) - 2)
            t = (p - c[k]) / (c[k + 1] - c[k])
            shape = [1, 1, 1]
            shape[2 - axis] = -1
            v0, v1 = v.index_select(2 - axis, k), v.index_select(2 - axis, k + 1)
            v = (v0 + t.reshape(shape) * (v1 - v0)) * inside.reshape(shape)
        return v.cpu().numpy()
    f = np.float32
    r, e = (torch.from_numpy(np.ascontiguousarray(a)).to(dev).double() for a in (s["ref"], s["ev"]))
    top = float(s["ref"].max())
    dta, dd, cut, far = float(f(0.1)), float(f(0.01 * top)), float(f(0.1 * top)), f(f(3.0) * f(0.1))
    sp = [f(v) for v in s["spacing"]]
    n = [int(f(far / v)) for v in sp]
    best = torch.full_like(r, float("inf"))
    nz, ny, nx = r.shape
    for k in range(-n[2], n[2] + 1):
        for j in range(-n[1], n[1] + 1):
            for i in range(-n[0], n[0] + 1):
                q = [f(sp[0] * f(i)), f(sp[1] * f(j)), f(sp[2] * f(k))]
                if f(f(f(q[0] * q[0]) + f(q[1] * q[1])) + f(q[2] * q[2])) > f(far * far):
                    continue
                d2 = sum((float(v) * m) ** 2 for v, m in zip(sp, (i, j, k)))
                here = (slice(max(0, -k), nz - max(0, k)), slice(max(0, -j), ny - max(0, j)), slice(max(0, -i), nx - max(0, i)))
                there = (slice(max(0, k), nz + min(0, k)), slice(max(0, j), ny + min(0, j)), slice(max(0, i), nx + min(0, i)))
                g = d2 / dta ** 2 + (e[there] - r[here]) ** 2 / dd ** 2
                best[here] = torch.minimum(best[here], g)
    g = torch.where(r >= cut, best.sqrt(), torch.full_like(best, -1.0))
    seen = r >= cut
    return g.cpu().numpy(), float((g[seen] <= 1.0).double().mean())
