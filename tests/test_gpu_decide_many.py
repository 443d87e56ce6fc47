"""Decisions that emit many copies per vertex: the time grows with the work, at every size of the
queue, and the one-cluster kernel's windows of copies give the oracle's queue."""
import numpy as np
import pytest

import nrrs_b200 as nb
import oracle as O
from gpu_util import empty, host, make_net, stream, torch_cuda

pytestmark = pytest.mark.gpu
MAXQ = 1 << 21


@pytest.fixture(scope="module")
def net():
    n = make_net()
    yield n
    n.close()


def best_us(net, n, copies, scale_up=1, clamp=250.0):
    """Microseconds per call of a decision with about `copies` copies of each of n vertices."""
    torch = torch_cuda()
    rng = np.random.default_rng(n)
    rrs = torch.from_numpy((1.0 if scale_up else copies) * rng.uniform(0.75, 1.0, n).astype(np.float32)).cuda()
    rnd = torch.from_numpy(rng.random(n, dtype=np.float32)).cuda()
    dp = nb.default_decide(scale_up=scale_up, clamp_max=clamp)
    cap = int(1.5 * copies * n) + 64
    norm, queue, size = empty(n), empty(cap, "int32"), empty(1, "int32")
    e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = float("inf")
    for _ in range(6):
        e0.record()
        for _ in range(20):
            net.decideEmit(rrs, rnd, n, int(2 * copies * n) if not scale_up else copies * n, 0, dp,
                           norm, None, queue, cap, size, stream=stream())
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) / 20 * 1e3)
    assert 0.8 * copies * n < int(size[0]) <= 1.1 * copies * n
    return best


# twice the vertices: at most twice the time (the launches do not double)
@pytest.mark.parametrize("n", [150_000, 200_000, 300_000])
def test_emission_time_grows_with_the_queue(net, n):
    assert best_us(net, n, 12) <= 2 * best_us(net, n // 2, 12)


# 65,536 vertices are one cluster's, one more is not: no jump where the kernels meet
@pytest.mark.parametrize("copies,scale_up,clamp", [(3, 0, 8.0), (7, 0, 8.0), (7, 1, 8.0), (12, 1, 250.0),
                                                   (50, 1, 250.0), (50, 0, 250.0)])
def test_cluster_no_slower_than_two_passes(net, copies, scale_up, clamp):
    assert best_us(net, 65_536, copies, scale_up, clamp) <= 1.2 * best_us(net, 65_537, copies, scale_up, clamp)


# windows of 10,240 copies: zeros, ones and long runs across their edges; on both sides of the rule
@pytest.mark.parametrize("n", [60, 4096, 4097, 8193, 30_001])
@pytest.mark.parametrize("kind", ["spread", "runs", "sidx", "overflow"])
@pytest.mark.parametrize("clamp", [8.0, 250.0])
def test_many_copies_against_oracle(net, n, kind, clamp):
    rng = np.random.default_rng(n)
    rrs = rng.uniform(0.05, clamp, n).astype(np.float32)
    if kind == "runs":
        rrs = np.where(rng.random(n) < 0.02, clamp, 0.05).astype(np.float32)
        rrs[n // 2:n // 2 + 50] = clamp
    rnd = rng.random(n, dtype=np.float32)
    dp = nb.default_decide(clamp_max=clamp)
    budget = int(np.ceil(rrs).sum())
    cap = budget // 3 if kind == "overflow" else 2 * budget + n
    sidx = rng.permutation(n).astype(np.uint32) if kind == "sidx" else None
    torch = torch_cuda()
    d_sidx = torch.from_numpy(sidx.view(np.int32)).cuda() if sidx is not None else None
    norm, queue, size, split = empty(n), empty(cap, "int32"), empty(1, "int32"), empty(n, "uint8")
    want = O.decide_emit(rrs, rnd, budget, 0, dp, capacity=cap, scatter_index=sidx, shift_n=MAXQ)
    for _ in range(2):
        queue.zero_()
        net.decideEmit(torch.from_numpy(rrs).cuda(), torch.from_numpy(rnd).cuda(), n, budget, 0, dp,
                       norm, split, queue, cap, size, scatter_index=d_sidx, stream=stream())
        _, flags = net.device_status(stream())
        total = int(host(size, np.uint32)[0])
        assert total == want["total"]
        assert np.array_equal(host(queue, np.uint32)[:min(total, cap)], want["queue"])
        assert np.array_equal(host(split)[:n], want["split"])
        assert bool(flags & nb.DEV_OVERFLOW) == (total > cap)
