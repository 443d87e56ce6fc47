"""Decisions that emit many copies per vertex: the time grows with the work, at every size of the
queue."""
import numpy as np
import pytest

import nrrs_b200 as nb
from gpu_util import empty, make_net, stream, torch_cuda

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
