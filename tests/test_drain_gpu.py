"""The drain kernel (small runs, and the end of every other one) against the
oracle, bit for bit, and against the waves in what it counts. Its edges: fewer
histories than warps, one more than a warp or than all warps' lanes hold, runs
just below and above the population at which it takes over, and a gradient
replay through it."""
import numpy as np
import pytest

from gegs_b200 import workloads as W

pytestmark = pytest.mark.gpu

WAVES = dict(photon_budget=32, electron_budget=4)      # a run that names its step budgets is run in waves


def _load(engine, job):
    sh = job.scene()
    engine.set_physics(job.physics)
    engine.set_scene(sh)
    return sh


@pytest.mark.parametrize("histories", [1, 31, 33, 3553, 4000, 4001, 20000, 70000])
@pytest.mark.parametrize("scene", ["slab", "head"])
def test_drain_is_the_oracle_and_counts_like_the_waves(engine, oracle, scene, histories):
    if scene == "slab":
        job = W.config2(histories=histories, nphsp=20000, n=30)
    else:
        job = W.config3(histories=histories, nphsp=20000, dims=(48, 40, 24), angles=(0.0, 72.0, 200.0))
    sh = _load(engine, job)
    drained = engine.run(0, histories)
    a = engine.tally()
    engine.reset_tally()
    waves = engine.run(0, histories, **WAVES)
    b = engine.tally()
    ref, _ = oracle.run(job.physics, sh, 0, histories)
    np.testing.assert_array_equal(a, ref)
    np.testing.assert_array_equal(b, ref)
    assert drained["error_bits"] == waves["error_bits"] == 0
    if histories <= 4000:
        assert drained["waves"] == 2                   # the plan before the drain kernel and the one after it
    for key in ("processed", "photon_steps", "electron_steps", "photon_steps_class", "electron_steps_class"):
        assert drained[key] == waves[key], key


def test_a_history_range_and_several_runs_on_one_engine(engine, oracle):
    """Drained runs of part of a plan, one after another and beside a run in
    waves, add up to the plan's tally."""
    job = W.config3(histories=9000, nphsp=5000, dims=(40, 40, 20))
    sh = _load(engine, job)
    for lo, hi, kw in ((0, 7, {}), (7, 3000, {}), (3000, 6001, WAVES), (6001, 9000, dict(batch=512))):
        engine.run(lo, hi, **kw)
    ref, _ = oracle.run(job.physics, sh, 0, 9000)
    np.testing.assert_array_equal(engine.tally(), ref)


def test_a_gradient_replay_drains_and_leaves_the_forward_run_as_it_was(engine):
    """The first run of an engine being a replay, then a forward run, then a
    replay again: the same gradient (double sums in any order) and the tally."""
    from gegs_b200.engine import Engine
    job = W.config4(histories=5000, nphsp=5000, dims=(40, 40, 20), nb=6, bixel=1.5)
    sh = _load(engine, job)
    g = np.random.default_rng(3).normal(size=sh.nvox)
    engine.run(0, 5000, **WAVES)
    want = engine.tally()
    fresh = Engine(0)
    fresh.set_physics(job.physics)
    fresh.set_scene(job.scene())
    first = fresh.backward(0, 5000, g)
    fresh.run(0, 5000)
    np.testing.assert_array_equal(fresh.tally(), want)
    again = fresh.backward(0, 5000, g)
    fresh.close()
    # sums of up to 1e6 products of both signs in double, in two orders: each is within 1e6 * 2^-53 = 1e-10
    # of the sum of its terms' sizes, some ten times the largest sum
    assert np.abs(first).max() > 0
    np.testing.assert_allclose(again, first, rtol=0, atol=1e-9 * np.abs(first).max())


COUNTS = ("processed", "photon_steps", "electron_steps", "photon_steps_class", "electron_steps_class")


def _split(job, n):
    """The plan with every bremsstrahlung photon split n ways."""
    job.physics = job.physics.copy()
    job.physics["nbr_split"] = n
    return job


@pytest.mark.parametrize("records", [0, 34, 1])
@pytest.mark.parametrize("scene,histories,split", [("slab", 4000, 1), ("slab", 20000, 1), ("slab", 3000, 100),
                                                   ("head", 3000, 1), ("head", 20000, 1), ("head", 400, 100)])
def test_full_stacks_go_on_in_waves(engine, oracle, scene, histories, split, records):
    """Stacks of the drain kernel that overflow, because photons are split more
    ways than a stack holds or because they are small: the tally is the oracle's,
    and the counts are those of a run in waves."""
    if scene == "slab":
        job = _split(W.config2(histories=histories, nphsp=20000, n=30), split)
    else:
        job = _split(W.config3(histories=histories, nphsp=20000, dims=(48, 40, 24), angles=(0.0, 72.0, 200.0)), split)
    sh = _load(engine, job)
    waves = engine.run(0, histories, **WAVES)
    engine.reset_tally()
    engine.set_drain_stack(records)
    try:
        drained = engine.run(0, histories)
    finally:
        engine.set_drain_stack(0)
    np.testing.assert_array_equal(engine.tally(), oracle.run(job.physics, sh, 0, histories)[0])
    assert drained["error_bits"] == 0
    if histories <= 4000:                              # the overflow is seen by the waves behind the drain kernel
        assert (drained["waves"] > 2) == (split == 100 or records == 1)
    for key in COUNTS:
        assert drained[key] == waves[key], key


def _tally_behind(engine, stream, nvox):
    """The tally as a copy queued on `stream` behind the launched run reads it,
    without waiting for the run."""
    import torch

    class View:
        __cuda_array_interface__ = dict(shape=(nvox,), typestr="<i8", data=(engine.tally_device_ptr(), False), version=3)
    with torch.cuda.stream(stream):
        out = torch.as_tensor(View(), device="cuda").clone()
    stream.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("histories", [3000, 20000])
def test_a_launched_run_is_whole_for_the_stream(engine, oracle, histories):
    """What full stacks left over is transported in the launch itself, not when
    the host waits for it: alone, and in a launch of several plans."""
    import torch
    from gegs_b200.engine import Engine, launch_group
    stream = torch.cuda.Stream()
    job = _split(W.config2(histories=histories, nphsp=5000, n=30), 100)
    sh = _load(engine, job)
    ref, _ = oracle.run(job.physics, sh, 0, histories)
    other = Engine(0)
    _load(other, job)
    engine.set_stream(stream)
    try:
        engine.launch(0, histories)
        np.testing.assert_array_equal(_tally_behind(engine, stream, sh.nvox), ref)
        assert engine.wait()["error_bits"] == 0
        engine.reset_tally()
        launch_group([engine, other], [(0, histories), (0, histories)])
        np.testing.assert_array_equal(_tally_behind(engine, stream, sh.nvox), ref)
        np.testing.assert_array_equal(_tally_behind(other, stream, sh.nvox), ref)
        engine.wait()
        other.wait()
    finally:
        engine.set_stream(None)
        other.close()


def test_a_gradient_replay_with_full_stacks(engine):
    job = W.config4(histories=5000, nphsp=5000, dims=(40, 40, 20), nb=6, bixel=1.5)
    sh = _load(engine, job)
    g = np.random.default_rng(3).normal(size=sh.nvox)
    for histories in (2000, 5000):
        want = engine.backward(0, histories, g)
        engine.set_drain_stack(20)
        try:
            got = engine.backward(0, histories, g)
        finally:
            engine.set_drain_stack(0)
        # double sums in another order, as above
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-9 * np.abs(want).max())


@pytest.mark.parametrize("turns", [1, 2, 40, 1000])
@pytest.mark.parametrize("scene,histories", [("slab", 1), ("slab", 4000), ("slab", 20000), ("head", 3553), ("head", 20000)])
def test_a_warp_out_of_turns_hands_its_particles_to_the_waves(engine, oracle, scene, histories, turns):
    """The drain kernel ends after a given number of turns whatever its particles
    do, also before a warp has claimed anything; the rest of the run is the
    waves', with the oracle's tally and the waves' counts."""
    if scene == "slab":
        job = W.config2(histories=histories, nphsp=20000, n=30)
    else:
        job = W.config3(histories=histories, nphsp=20000, dims=(48, 40, 24), angles=(0.0, 72.0, 200.0))
    sh = _load(engine, job)
    waves = engine.run(0, histories, **WAVES)
    ref, _ = oracle.run(job.physics, sh, 0, histories)
    engine.set_drain_turns(turns)
    try:
        for kw in ({}, dict(batch=600)):
            engine.reset_tally()
            drained = engine.run(0, histories, **kw)
            np.testing.assert_array_equal(engine.tally(), ref)
            assert drained["error_bits"] == 0
            for key in COUNTS:
                assert drained[key] == waves[key], key
            if histories <= 4000 and not kw and turns <= (2 if histories == 1 else 40):
                assert drained["waves"] > 2
    finally:
        engine.set_drain_turns(0)


@pytest.mark.parametrize("kw", [{}, dict(photon_budget=16), dict(pipelined=False), dict(max_waves=10), dict(batch=1),
                                dict(mode=1), dict(mode=2)])
def test_an_empty_range_is_a_run_of_nothing(kw):
    """The first run of an engine, with the drain kernel and without."""
    from gegs_b200.engine import Engine
    e = Engine(0)
    sh = _load(e, W.config1(histories=100, n=10, voxel=3.0))
    for h in (0, 50):
        st = e.run(h, h, **kw)
        assert st["error_bits"] == 0 and sum(st["processed"]) == 0
    assert not e.tally().any()
    e.close()


def test_without_memory_for_the_stacks_a_run_goes_in_waves(oracle):
    """The queues are there already, and less memory is free than the stacks take (225 MB)."""
    import torch
    from gegs_b200.engine import Engine
    job = W.config3(histories=3000, nphsp=5000, dims=(40, 40, 20))
    loaded, e = Engine(0), Engine(0)
    _load(loaded, job)
    loaded.run(0, 3000)                               # the kernels' own memory
    loaded.close()
    sh = _load(e, job)
    ref, _ = oracle.run(job.physics, sh, 0, 3000)
    opts = dict(batch=1 << 16)
    e.run(0, 3000, **opts, **WAVES)
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info(0)[0] - (180 << 20), dtype=torch.uint8, device="cuda")
    for last in (False, True):
        for _ in range(2):
            e.reset_tally()
            st = e.run(0, 3000, **opts)
            np.testing.assert_array_equal(e.tally(), ref)
            assert (st["waves"] == 2) == last
        held = None
        torch.cuda.empty_cache()
    e.close()


@pytest.mark.parametrize("kw", [dict(photon_budget=2, electron_budget=1), dict(pipelined=False), dict(max_waves=1000),
                                dict(pipelined=False, photon_budget=3, stage_tables=True), {}])
def test_drain_and_no_drain_by_name(engine, oracle, kw):
    """Beside every option that otherwise decides it, both ways, alone and launched."""
    from gegs_b200.engine import launch_group
    for histories in (3000, 9000):
        job = W.config3(histories=histories, nphsp=20000, dims=(48, 40, 24), angles=(0.0, 72.0, 200.0))
        sh = _load(engine, job)
        ref, _ = oracle.run(job.physics, sh, 0, histories)
        small = histories <= 4000
        for drain in (True, False):
            engine.reset_tally()
            st = engine.run(0, histories, drain=drain, **kw)
            np.testing.assert_array_equal(engine.tally(), ref)
            assert (st["waves"] == 2) == (drain and small)
            if "max_waves" in kw:
                continue                               # not an option of launched runs
            engine.reset_tally()
            engine.launch(0, histories, drain=drain, **kw)
            assert (engine.wait()["waves"] == 2) == (drain and small)
            np.testing.assert_array_equal(engine.tally(), ref)
            engine.reset_tally()
            launch_group([engine], [(0, histories)], [dict(drain=drain, **kw)])
            assert (engine.wait()["waves"] == 2) == (drain and small)
            np.testing.assert_array_equal(engine.tally(), ref)


def test_a_particle_that_does_not_end_uses_up_the_waves(engine):
    """What the drain kernel hands over comes under the wave budget: with two
    turns a warp and six waves, an ordinary plan is such a one."""
    from gegs_b200.engine import GegsError
    job = W.config2(histories=2000, nphsp=2000, n=30)
    _load(engine, job)
    engine.set_drain_turns(2)
    try:
        with pytest.raises(GegsError) as err:
            engine.run(0, 2000, max_waves=6, drain=True)
    finally:
        engine.set_drain_turns(0)
    assert err.value.status == 6                      # GEGS_ERR_STEP_BUDGET
    assert engine.stats()["waves"] == 6


@pytest.mark.parametrize("phantom_first", [False, True])
def test_without_memory_for_the_kernels_own_frames_a_run_goes_in_waves(phantom_first):
    """A process whose first run of the drain kernel would find room for the stacks
    (228 MB), but not for the frames of its threads (190 MB more): it must not be
    launched. With `phantom_first` the engine has drained a plan without jaws and
    MLC, whose kernel has smaller frames."""
    import os
    import subprocess
    import sys
    code = f"phantom_first = {phantom_first}" + """
import numpy as np, torch
from gegs_b200 import workloads as W
from gegs_b200.engine import Engine
job = W.config3(histories=3000, nphsp=5000, dims=(40, 40, 20))
e = Engine(0)
if phantom_first:
    slab = W.config2(histories=1000, nphsp=1000, n=20)
    e.set_physics(slab.physics)
    e.set_scene(slab.scene())
    assert e.run(0, 1000, batch=1 << 16)["waves"] == 2
e.set_physics(job.physics)
e.set_scene(job.scene())
e.run(0, 3000, batch=1 << 16, drain=False)
want = e.tally()
held = torch.empty(torch.cuda.mem_get_info(0)[0] - (300 << 20), dtype=torch.uint8, device="cuda")
for last in (False, True):
    for _ in range(2):
        e.reset_tally()
        st = e.run(0, 3000, batch=1 << 16)
        np.testing.assert_array_equal(e.tally(), want)
        assert (st["waves"] == 2) == last, st["waves"]
    held = None
    torch.cuda.empty_cache()
e.close()
print("as it should be")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, PYTHONPATH=root), capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "as it should be" in r.stdout, r.stdout + r.stderr
