"""Decisions on factors that no inference gives (negative, infinite, NaN): the one-cluster kernel makes
of them what the two passes make, in bounded time and within the queue. A count is the factor's
integer part as an unsigned number; the next size is the sum of the 2,048-vertex chunks' totals
(saturating), and a chunk emits its split bytes from its prefix on. (Where a wrapped total lets two
chunks write the same entries, either may come last.)"""
import numpy as np
import pytest

import nrrs_b200 as nb
from gpu_util import empty, host, make_net, stream, torch_cuda

pytestmark = pytest.mark.gpu
ODD = np.float32([np.nan, np.inf, -np.inf, -1.0, -1.5, -3.0, -300.0, -3.4e38, -0.5, -0.0, 300.0, 255.5])


@pytest.fixture(scope="module")
def net():
    n = make_net(max_queue=1 << 18, max_train=256)
    yield n
    n.close()


def expected(rrs, rnd, cap):
    """Split bytes, queue and next size of factors that are not scaled."""
    n = len(rrs)
    with np.errstate(invalid="ignore"):
        big = ~(rrs < 256)
        part = np.where(np.isfinite(rrs) & ~big, np.trunc(rrs), 0)
        s = np.clip(part, -2.0 ** 31, 255).astype(np.int64)
        s = np.where(np.isneginf(rrs), -2 ** 31, s)
        frac = (rrs - s.astype(np.float32)).astype(np.float32)
        s = np.where(rnd <= frac, s + 1, s)
    s = np.where(big, 255, np.minimum(s, 255))
    s = np.where(np.isnan(rrs), 0, s) & 0xffffffff
    # a run of 8 vertices is stored in words: the upper bytes of a count fall on its neighbours
    b = (s & 255).astype(np.uint8)
    for v in range(0, n - n % 8, 4):
        word = 0
        for j in range(4):
            word |= int(s[v + j]) << (8 * j) & 0xffffffff
        b[v:v + 4] = [word >> (8 * j) & 255 for j in range(4)]
    queue, wrote, size = np.zeros(cap, np.uint32), np.zeros(cap, np.int64), 0
    for c in range(0, n, 2048):
        ids = np.repeat(np.arange(c, min(n, c + 2048), dtype=np.uint32), b[c:c + 2048])
        at = min(size, 0xffffffff)
        k = max(0, min(len(ids), cap - at))
        queue[at:at + k] = ids[:k]
        wrote[at:at + k] += 1
        size += int(s[c:c + 2048].sum()) & 0xffffffff
    return b, queue, wrote, min(size, 0xffffffff)


@pytest.mark.parametrize("n", [33, 2048, 5000, 8193, 30_001, 65_536, 70_000])
@pytest.mark.parametrize("few", [True, False])
def test_odd_factors(net, n, few):
    torch = torch_cuda()
    rng = np.random.default_rng(n)
    rrs = rng.uniform(0.0, 8.0, n).astype(np.float32)
    m = rng.choice(n, 3, replace=False) if few else np.flatnonzero(rng.random(n) < 0.2)
    rrs[m] = [-1.0, -np.inf, -1.5] if few else rng.choice(ODD, len(m))
    rnd = rng.uniform(0.01, 0.99, n).astype(np.float32)
    cap = 9 * n
    # the sum that scales stays positive and below the budget: a scale of 1
    rrs[:16] = 8.0
    d_rrs, d_rnd = torch.from_numpy(rrs).cuda(), torch.from_numpy(rnd).cuda()
    sum_acc = torch.ones(1, dtype=torch.int64, device="cuda")
    norm, split, queue, size = empty(n), empty(n, "uint8"), empty(cap, "int32"), empty(1, "int32")
    net.decideEmitWithSum(d_rrs, d_rnd, n, 1 << 30, 0, sum_acc, nb.default_decide(), norm, split,
                          queue, cap, size, stream=stream())
    net.device_status(stream())
    b, want, wrote, total = expected(rrs, rnd, cap)
    assert int(host(size, np.uint32)[0]) == total
    assert np.array_equal(host(split)[:n], b)
    got = host(queue, np.uint32)[:cap]
    assert np.array_equal(got[wrote == 1], want[wrote == 1])
    assert not got[wrote == 0].any()


# the allocation-free entry point, on finite factors (its own sum scales: positive, below the budget)
@pytest.mark.parametrize("n", [33, 2048, 5000, 30_001, 70_000])
def test_odd_factors_noalloc(n):
    torch = torch_cuda()
    rng = np.random.default_rng(n)
    rrs = rng.uniform(0.5, 8.0, n).astype(np.float32)
    rrs[rng.choice(n, 5, replace=False)] = [-1.0, -1.5, -3.0, -7.25, -0.5]
    rnd = rng.uniform(0.01, 0.99, n).astype(np.float32)
    cap = 9 * n
    norm, split, queue, size = empty(n), empty(n, "uint8"), empty(cap, "int32"), empty(1, "int32")
    nb.decide_emit_noalloc(torch.from_numpy(rrs).cuda(), torch.from_numpy(rnd).cuda(), n, 1 << 30, 0,
                           nb.default_decide(), norm, split, queue, cap, size, stream=stream())
    nb.noalloc_device_status(stream())
    b, want, wrote, total = expected(rrs, rnd, cap)
    assert int(host(size, np.uint32)[0]) == total
    assert np.array_equal(host(split)[:n], b)
    got = host(queue, np.uint32)[:cap]
    assert np.array_equal(got[wrote == 1], want[wrote == 1])
    assert not got[wrote == 0].any()
