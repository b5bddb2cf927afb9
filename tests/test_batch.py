"""Several plans at once on one GPU: each plan's tally equals its own run,
bit for bit, whether the plans run concurrently or one after another."""
import numpy as np
import pytest

from gegs_b200 import workloads as W
from gegs_b200.batch import choose_options


def test_choose_options_respects_memory_share():
    o = choose_options(100_000_000, 64e9)
    assert o["batch"] == 1 << 22 and o["refill_below"] == o["batch"] // 4
    small = choose_options(10_000, 64e9)
    assert small["batch"] == 1 << 16
    capped = choose_options(100_000_000, 1e9)
    assert capped["batch"] * 4.5e3 <= 1e9 and capped["batch"] >= 1 << 16


@pytest.mark.gpu
def test_concurrent_plans_match_their_own_runs(oracle):
    from gegs_b200.batch import PlanBatch
    jobs = W.config5(n_plans=4, hist_min=2000, hist_max=20000, nphsp=5000, dims_max=(48, 48, 32), dims_min=24)
    pb = PlanBatch(jobs, memory_budget_gb=4.0)
    st = pb.run()
    conc = pb.tallies()
    pb.run_sequential()
    seq = pb.tallies()
    for a, b, s in zip(conc, seq, st):
        np.testing.assert_array_equal(a, b)
        assert s["error_bits"] == 0 and a.sum() > 0
    ref, _ = oracle.run(jobs[1].physics, jobs[1].scene(), 0, jobs[1].histories)
    np.testing.assert_array_equal(conc[1], ref)
    pb.close()


def test_launch_group_checks_its_arguments():
    from gegs_b200.engine import launch_group
    with pytest.raises(ValueError):
        launch_group([], [])
    with pytest.raises(ValueError):
        launch_group([object()], [(0, 1), (1, 2)])


@pytest.mark.gpu
def test_one_launch_equals_launches_per_plan_and_the_oracle(oracle):
    """All plans as one graph launch (a branch per plan, gegs_launch_group):
    each plan's tally equals its launch on its own stream and the oracle; the
    group refuses an engine twice and an engine with a run in flight."""
    from gegs_b200.batch import PlanBatch
    from gegs_b200.engine import GegsError, launch_group
    jobs = W.config5(n_plans=5, hist_min=2000, hist_max=20000, nphsp=5000, dims_max=(48, 48, 32), dims_min=24)
    pb = PlanBatch(jobs, memory_budget_gb=4.0)
    st = pb.run(one_launch=True)
    one = pb.tallies()
    pb.run(one_launch=True)                                          # the cached group graph again
    again = pb.tallies()
    pb.run(one_launch=False)
    per = pb.tallies()
    for a, b in zip(one, again):
        np.testing.assert_array_equal(a, b)
    for a, b, s in zip(one, per, st):
        np.testing.assert_array_equal(a, b)
        assert s["error_bits"] == 0 and a.sum() > 0 and s["waves"] > 0
    for k in (0, 3):
        ref, _ = oracle.run(jobs[k].physics, jobs[k].scene(), 0, jobs[k].histories)
        np.testing.assert_array_equal(one[k], ref)
    e = pb.engines
    with pytest.raises(GegsError):
        launch_group([e[0], e[1], e[0]], [(0, 10)] * 3)
    e[2].launch(0, 10)
    with pytest.raises(GegsError):
        launch_group([e[1], e[2]], [(0, 10)] * 2)
    e[2].wait()
    launch_group(e[:2], [(0, 100), (0, 100)])                       # the engines are usable again
    for x in e[:2]:
        x.wait()
    pb.close()


@pytest.mark.gpu
def test_autotuned_plans_keep_their_tallies(oracle):
    """The autotuner changes only how a plan runs (batch, grid, step budgets,
    refill threshold): every candidate it times gives the same tally, and the
    plan tuned by it still equals the oracle bit for bit."""
    from gegs_b200.batch import PlanBatch, autotune
    from gegs_b200.engine import Engine
    job = W.config3(histories=6000, nphsp=4000, dims=(40, 40, 24))
    e = Engine(0)
    e.set_physics(job.physics)
    e.set_scene(job.scene())
    best, best_ms, trials = autotune(e, job, sample=3000)
    assert len(trials) >= 8 and best_ms == min(t for _, t in trials)
    seen = set()
    for o, _ in trials:
        e.reset_tally()
        e.run(0, 3000, **o)
        seen.add(e.tally().tobytes())
    assert len(seen) == 1
    e.close()
    pb = PlanBatch([job], memory_budget_gb=2.0, tune_sample=2000)
    pb.run()
    ref, _ = oracle.run(job.physics, job.scene(), 0, job.histories)
    np.testing.assert_array_equal(pb.tallies()[0], ref)
    pb.close()


@pytest.mark.parametrize("histories", [10_000, 300_000, 5_000_000, 100_000_000])
def test_a_plans_memory_stays_within_its_share(histories):
    """Queues and drain stacks together, down to the smallest batch's queues."""
    stacks = 3552 * (14 * 64 * 64 + 3 * 64 * 32)        # warps of the drain kernel x records, on the B200
    for share in (1e8, 3.5e8, 5.6e8, 5.8e8, 6.25e8, 7e8, 9e8, 1.4e9, 3e9, 6e9, 2.2e10, 4e10):
        o = choose_options(histories, share)
        used = o["batch"] * 5.2e3 + (stacks if o["drain"] else 0)
        assert used <= max(share, (1 << 16) * 5.2e3), (share, o)
        assert o["drain"] == (share >= 5.8e8)           # where both fit


@pytest.mark.gpu
def test_a_batch_of_plans_stays_within_its_budget():
    import torch
    from gegs_b200.batch import PlanBatch
    jobs = [W.config1(histories=300_000, n=10, voxel=3.0) for _ in range(8)]
    warm = PlanBatch(jobs[:1], memory_budget_gb=1.0)     # the kernels' own memory
    warm.run([1000])
    warm.close()
    for budget in (8 * 0.7, 8 * 0.4):
        before = torch.cuda.mem_get_info(0)[0]
        pb = PlanBatch(jobs, memory_budget_gb=budget)
        stats = pb.run([2000] * 8)
        used = before - torch.cuda.mem_get_info(0)[0]
        pb.close()
        assert all((s["waves"] == 2) == (budget > 5) for s in stats)   # drained where the stacks fit
        assert used < budget * 1e9 + 8 * 30e6            # tables (5 MB), scene and graph of a plan besides


class _Timed:
    """An engine whose runs take a made-up time: every other one is the fastest so far."""
    def __init__(self):
        self.runs = []

    def run(self, h0, h1, **o):
        self.runs.append(o)
        return dict(device_ms=1000.0 - len(self.runs) if len(self.runs) % 4 else 2000.0)

    def reset_tally(self):
        pass


@pytest.mark.parametrize("start", [None, dict(batch=1 << 17), dict(batch=1 << 17, photon_budget=8)])
def test_the_autotuner_changes_one_thing_at_a_time(start):
    """Whether a plan's end goes to the drain kernel is a dimension of its own:
    a trial of a step budget or of the wave order says so by name, and does not
    switch it by the way."""
    from gegs_b200.batch import autotune
    job = W.config1(histories=5000, n=8, voxel=3.0)
    e = _Timed()
    best, best_ms, trials = autotune(e, job, start=start)
    assert {o["drain"] for o, _ in trials} == {True, False}
    assert trials[0][0]["drain"] == (start is None or "photon_budget" not in start)
    base, t0 = trials[0]
    for o, t in trials[1:]:
        d = {k for k in set(o) | set(base) if o.get(k) != base.get(k)}
        assert len(d - {"refill_below"}) == 1 or d == {"refill_below"}, (base, o)
        if t < t0:
            base, t0 = o, t
    assert (best, best_ms) == (base, t0)
