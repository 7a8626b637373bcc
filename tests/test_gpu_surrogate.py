"""The surrogate network's paths that depend on how many rows a call has: predictions in
groups of batches, in two slots, against the same rows batch by batch (tolerance: none, a
group's products are summed as a batch's) and against the CPU reference (the tolerance of a
forward pass in bfloat16 operands, 1e-2 as for one batch); gradients at ragged sizes, with
products of few and of many blocks; and training steps whose recorded forms are made, kept
and dropped again as sizes come and go (tolerance: none)."""
import numpy as np
import pytest

import surrogate_ref as ref

pytestmark = pytest.mark.gpu


def _case(n, seed):
    rng = np.random.default_rng(seed)
    flat = (ref.init_params(seed) + rng.normal(0.0, 0.02, ref.init_params(seed).shape)).astype(np.float32)
    return flat, rng.random((n, ref.N_IN)).astype(np.float32), rng.normal(0.0, 1.0, (n, ref.T_OUT, ref.N_OUT)).astype(np.float32)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("max_batch,n", [(64, 1), (64, 65), (64, 2048), (64, 4200), (200, 2047), (200, 5121), (2100, 2200)])
def test_predictions_in_groups_are_those_of_single_batches(max_batch, n):
    from covidsim_b200 import surrogate
    flat, x, _ = _case(n, 21)
    net = surrogate.Surrogate(max_batch=max_batch, params=flat)
    step = (max_batch + 63) // 64 * 64                 # the capacity that the batch is rounded up to
    single = np.concatenate([net.predict(x[i:i + step]) for i in range(0, n, step)])
    for _ in range(2):                                 # the second call finds the workspace in place
        assert np.array_equal(net.predict(x), single)
    pick = np.unique(np.linspace(0, n - 1, 40).astype(int))
    assert _rel(single[pick], ref.forward(flat, x[pick], round_bf16=True)) < 1e-2
    net.set_gemm("mma.sync")                           # one batch at a time; only summation order differs
    assert _rel(net.predict(x), single) < 2e-3
    net.close()


@pytest.mark.parametrize("n", [1, 63, 129, 300])
def test_gradients_at_ragged_sizes(n):
    from covidsim_b200 import surrogate
    flat, x, target = _case(n, 23)
    out = {}
    for impl in ("tcgen05", "mma.sync"):
        net = surrogate.Surrogate(max_batch=320, params=flat)
        net.set_gemm(impl)
        out[impl] = net.loss_grad(x, target)
        again = net.loss_grad(x, target)
        assert again[0] == out[impl][0] and np.array_equal(again[1], out[impl][1])
        net.close()
    assert abs(out["tcgen05"][0] - out["mma.sync"][0]) <= 1e-4 * abs(out["mma.sync"][0])
    k = 0
    for name, (o, i) in ref.layer_shapes():
        for part, m in (("W", o * i), ("b", o)):
            e = _rel(out["tcgen05"][1][k:k + m], out["mma.sync"][1][k:k + m])
            assert e < 1e-2, (name, part, e)
            k += m


def test_training_steps_do_not_depend_on_what_is_recorded():
    from covidsim_b200 import surrogate
    flat, x, target = _case(200, 25)
    sizes = [200, 1, 64, 65, 100, 127, 128, 129, 190, 7, 200, 1, 64, 100]   # ten sizes, then some again
    a, b = (surrogate.Surrogate(max_batch=256, params=flat) for _ in range(2))
    for k, n in enumerate(sizes):
        la = a.train_step(x[:n], target[:n], 1e-3)
        if k % 2:
            b.loss_grad(x[:n + 3], target[:n + 3]) if n + 3 <= 200 else b.predict(x)
        lb = b.train_step(x[:n], target[:n], 1e-3)
        assert la == lb, (k, n)
        assert np.array_equal(a.get_params(), b.get_params()), (k, n)
    a.close()
    b.close()


def test_many_batch_sizes_in_turn_do_not_record_at_every_step():
    """Twelve sizes in turn: once as many as are kept have been recorded, the others run
    without, and all give the steps of a network that sees them for the first time."""
    import torch
    from torch.profiler import profile, ProfilerActivity
    from covidsim_b200 import surrogate
    flat, x, target = _case(200, 27)
    net = surrogate.Surrogate(max_batch=256, params=flat)
    sizes = [200 - 16 * k for k in range(12)]

    def cycle():
        return [net.train_step(x[:n], target[:n], 1e-3) for n in sizes]
    cycle()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        cycle()
        cycle()
    names = [e.name for e in p.events()]
    if not names:
        pytest.skip("the profiler records nothing here")
    assert sum("GraphLaunch" in n for n in names) > 0
    assert sum("GraphInstantiate" in n for n in names) == 0
    fresh = surrogate.Surrogate(max_batch=256, params=net.get_params())
    for n in sizes:
        a, b = net.loss_grad(x[:n], target[:n]), fresh.loss_grad(x[:n], target[:n])
        assert a[0] == b[0] and np.array_equal(a[1], b[1]), n
    # sizes that are met from now on take the places of those that are not
    for n in sizes[:2] * 200:
        net.train_step(x[:n + 1], target[:n + 1], 1e-3)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        for n in sizes[:2]:
            net.train_step(x[:n + 1], target[:n + 1], 1e-3)
    assert sum("GraphLaunch" in e.name for e in p.events()) == 2
    net.close()
    fresh.close()
    torch.cuda.synchronize()


def test_memory_of_a_network_by_its_batch():
    """Activations, their gradients, scratch and batch of one row: 1.30 MB at most, so that the
    largest batch that fits the device does not shrink."""
    import torch
    from covidsim_b200 import surrogate
    torch.cuda.synchronize()
    used = {}
    for rows in (1024, 4096):
        free = torch.cuda.mem_get_info()[0]
        net = surrogate.Surrogate(max_batch=rows)
        used[rows] = free - torch.cuda.mem_get_info()[0]
        net.close()
    assert (used[4096] - used[1024]) / 3072 < 1.30e6


def test_a_network_takes_few_allocations():
    """No more than the 36 arrays it had when its passes ran in one chain: each allocation is
    host time of every creation."""
    from torch.profiler import profile, ProfilerActivity
    from covidsim_b200 import surrogate
    flat = ref.init_params(3).astype(np.float32)
    surrogate.Surrogate(max_batch=64, params=flat).close()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        net = surrogate.Surrogate(max_batch=64, params=flat)
    names = [e.name for e in p.events()]
    net.close()
    if not names:
        pytest.skip("the profiler records nothing here")
    assert 0 < sum(n == "cudaMalloc" for n in names) <= 36
