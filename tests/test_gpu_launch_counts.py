"""The count of kernels launched (cs_gpu_launch_count), and the names that per-launch timing
gives them, against the kernels that the profiler sees: direct calls, timesteps as graphs, the
run loop as day graphs (with parts that run on few days), without graphs and with timing
nodes, and a batch of one."""
import os
import re
import sys

import pytest

from covidsim_b200 import abi, sim
from tests.helpers import tiny_world

pytestmark = pytest.mark.gpu


def _kernels(f):
    """The library's kernels that ran on the device during f()."""
    import torch
    from torch.profiler import profile, ProfilerActivity
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
        f()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("the profiler records nothing here")
    return [n for n in names if re.match(r"(void )?k_\w+([(<]|$)", n)]


def _counted(s, f):
    n0 = s.backend.launches()
    seen = _kernels(f)
    return s.backend.launches() - n0, len(seen)


@pytest.mark.parametrize("fpr", [0.0, 0.1])
@pytest.mark.parametrize("form", ["graphs", "eager", "timed"])
@pytest.mark.parametrize("every_step", [False, True])
def test_launch_count_of_a_run(form, every_step, fpr):
    pop, P, lk, hr = tiny_world(adunit_grid=2)
    q = abi.cs_params.from_buffer_copy(P)
    q.FalsePositiveRate = fpr
    s = sim.Simulation(pop, q, lk, hr)
    if form == "eager":
        s.backend.lib.cs_gpu_use_graphs(s.backend.ctx, 0)
    if form == "timed":
        s.backend.profile(1)
    policy = sim.InterventionPolicy(threshold=3, window=7, duration=12.0)
    run = lambda: s.run(505, 40, n_seed=20, policy=policy, probs_every_step=every_step)   # noqa: E731
    run()   # graphs captured
    counted, seen = _counted(s, run)
    assert counted == seen > 40 * 4 * 9
    names = set(s.backend.profile_entries()) if form == "timed" else set()
    assert all(re.fullmatch(r"k_\w+(<\w+(, ?\w+)*>)?", n) for n in names), names
    if names:
        assert {"k_scan", "k_moves", "k_household", "k_day_check"} <= {n.split("<")[0] for n in names}
    s.close()


@pytest.mark.parametrize("fpr", [0.0, 0.1])
def test_launch_count_of_timesteps_sweeps_and_a_batch(fpr):
    pop, P, lk, hr = tiny_world()
    q = abi.cs_params.from_buffer_copy(P)
    q.FalsePositiveRate = fpr
    s = sim.Simulation(pop, q, lk, hr)
    seeds, dt = s.choose_seeds(5, 50), P.ModelTimeStep

    def steps():
        s.backend.begin_run(5, seeds)
        for k in range(6):
            s.backend.step(k * dt)
        s.backend.update_probs(0)
        s.backend.infect_sweep(6 * dt)
        s.backend.incub_recovery_sweep(6 * dt)
        s.backend.sync()
    steps()
    counted, seen = _counted(s, steps)
    assert counted == seen
    batch = sim.Batch([s])

    def batched():
        s.backend.begin_run(5, seeds)
        for k in range(6):
            batch.step(k * dt)
        batch.sync()
    batched()
    counted, seen = _counted(s, batched)
    assert counted == seen
    run = lambda: batch.run([5], 40, n_seed=20, policy=sim.InterventionPolicy(threshold=3, window=7, duration=12.0))   # noqa: E731
    run()
    counted, seen = _counted(s, run)
    assert counted == seen
    batch.close()
    s.close()


def test_timed_kernels_have_their_bytes_in_the_benchmark():
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import bench
    pop, P, lk, hr = tiny_world()
    s = sim.Simulation(pop, P, lk, hr)
    s.backend.profile(1)
    s.run(5, 20, n_seed=200)
    w = abi.counters_to_dict(s.backend.counters())
    names = {n.split("<")[0] for n in s.backend.profile_entries()}
    for k in ("k_scan", "k_household", "k_places", "k_spatial", "k_infections", "k_onsets", "k_progress", "k_moves"):
        assert k in names and bench.kernel_bytes(k, w, pop.n_cells * 80) > 0, k
    s.close()


def test_timed_names_are_the_kernels_that_run():
    pop, P, lk, hr = tiny_world(adunit_grid=2)
    s = sim.Simulation(pop, P, lk, hr)
    s.backend.profile(1)

    def work():
        s.run(505, 40, n_seed=20, policy=sim.InterventionPolicy(threshold=3, window=7, duration=12.0))
        s.backend.update_probs(0)
        s.backend.infect_sweep(40.0)
        s.backend.incub_recovery_sweep(40.0)
    ran = {re.search(r"k_\w+", n).group() for n in _kernels(work)}
    timed = {n.split("<")[0] for n in s.backend.profile_entries()}
    assert timed and timed <= ran, timed - ran
    s.close()
