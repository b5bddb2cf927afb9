"""Copies of ordinary host memory through the pinned buffers, at the sizes where a
chunk or a thread's share begins and ends, alone and from several threads at
once; and the device's largest reference dose behind the global gamma."""
import threading

import numpy as np
import pytest

from gegs_b200 import workloads as W

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("nbytes", [8, 2 * MB - 8, 2 * MB, 2 * MB + 8, 8 * MB - 8, 8 * MB + 8, 17 * MB + 16])
def test_a_tally_goes_out_and_comes_back_unchanged(engine, nbytes):
    n = nbytes // 8
    job = W.config1(histories=10, n=2, voxel=3.0)
    p = job.phantom
    p["x_bounds"] = np.arange(n + 1, dtype=np.float32)            # n voxels in a row
    p["y_bounds"] = p["z_bounds"] = np.float32([0.0, 1.0])
    p["voxel_med"], p["voxel_rhof"] = np.zeros(n, np.uint16), np.ones(n, np.float32)
    engine.set_physics(job.physics)
    engine.set_scene(job.scene())
    t = np.random.default_rng(n).integers(-2**60, 2**60, n)
    engine.set_tally(t)
    np.testing.assert_array_equal(engine.tally(), t)
    mass = np.random.default_rng(1).uniform(0.5, 2.0, n).astype(np.float32)
    want = t.astype(np.float64) * 2.0 ** -30 / mass.astype(np.float64) * 1.6e-8
    np.testing.assert_array_equal(engine.dose(mass), want)


def test_several_threads_at_once():
    """Six at once: more than the sets of buffers, so some take the driver's way."""
    from gegs_b200.postprocess import ct_ramp
    rng = np.random.default_rng(4)
    media = ["AIR700ICRU", "LUNG700ICRU", "ICRUTISSUE700ICRU", "ICRPBONE700ICRU"]
    seg = [(media.index(n), ub, lo, hi) for n, ub, lo, hi in W.CT_RAMP]
    hu = [rng.integers(-1100, 2600, 3_000_000 + 77 * k).astype(np.int16) for k in range(6)]
    got = [None] * 6

    def work(k):
        for _ in range(3):
            got[k] = ct_ramp(hu[k], seg, W.CT_LOWER)
    t = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [x.start() for x in t]
    [x.join() for x in t]
    for k in range(6):
        med, dens = W.hu_to_material(hu[k], media)
        np.testing.assert_array_equal(got[k][0], med)
        np.testing.assert_array_equal(got[k][1], dens)
    from gegs_b200.engine import load_library
    load_library().gegs_trim()
    np.testing.assert_array_equal(ct_ramp(hu[0], seg, W.CT_LOWER)[0], got[0][0])


@pytest.mark.parametrize("shape,top", [((3, 5, 7), 2.5), ((40, 33, 29), 0.003), ((2, 2, 2), 1e30)])
def test_gamma_is_relative_to_the_largest_reference_dose(shape, top):
    import ctypes as C
    from gegs_b200.postprocess import _lib, gamma3d
    rng = np.random.default_rng(6)
    ref = (rng.uniform(-0.2, 0.9, shape) * top).astype(np.float32)
    ref[tuple(s // 2 for s in shape)] = np.float32(top)
    ev = (ref * rng.normal(1.0, 0.02, shape)).astype(np.float32)
    g, rate = gamma3d(ref, ev, (0.1, 0.1, 0.25))
    m = float(ref.max())
    want = np.empty(ref.size, np.float32)
    ne, npass = C.c_uint64(), C.c_uint64()
    nz, ny, nx = shape
    assert _lib().gegs_gamma3d(0, ref.ctypes.data, ev.ctypes.data, nx, ny, nz, 0.1, 0.1, 0.25, 0.1, 0.01 * m, 0.1 * m, 3.0,
                               want.ctypes.data, C.byref(ne), C.byref(npass)) == 0
    np.testing.assert_array_equal(g.reshape(-1), want)
    assert rate == npass.value / ne.value
    for bad in (np.full(shape, np.nan, np.float32), -np.abs(ref)):
        with pytest.raises(RuntimeError):
            gamma3d(bad, ev, (0.1, 0.1, 0.25))
    one = ref.copy()
    one[0, 0, 0] = np.nan
    with pytest.raises(RuntimeError):
        gamma3d(one, ev, (0.1, 0.1, 0.25))
