"""The one-cluster decision of short queues (up to 65,536 vertices, 8,192 per CTA) at its edges,
against the oracle bit for bit: CTA and cluster boundaries, more entries than the stage holds, no
split array, scattered and misaligned arrays, a full queue, and repeated calls."""
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


@pytest.mark.parametrize("n", [1, 7, 9, 8191, 8192, 8193, 16385, 24577, 32768, 65535, 65536, 65537])
@pytest.mark.parametrize("kind", ["plain", "full_split", "sidx_off1", "overflow"])
def test_short_queue(net, n, kind):
    torch = torch_cuda()
    rng = np.random.default_rng(n)
    dp = nb.default_decide(scale_up=1) if kind == "full_split" else nb.default_decide()
    rrs = np.clip(rng.lognormal(-0.3, 1.2, n), 0.05, 8).astype(np.float32)
    rnd = rng.random(n, dtype=np.float32)
    # a large budget with scale_up: about 5 copies of every vertex, past the CTA's stage
    budget = 5 * n if kind == "full_split" else n
    cap = n // 2 if kind == "overflow" else 12 * n + 8
    sidx = rng.permutation(n).astype(np.uint32) if kind == "sidx_off1" else None
    off = 1 if kind == "sidx_off1" else 0
    pad = lambda a: torch.from_numpy(np.concatenate([np.zeros(off, a.dtype), a])).cuda()  # noqa: E731
    d_rrs, d_rnd = pad(rrs), pad(rnd)
    d_sidx = torch.from_numpy(sidx.view(np.int32)).cuda() if sidx is not None else None
    d_norm, d_queue, d_size = empty(n + off), empty(cap, "int32"), empty(1, "int32")
    d_split = empty(n + off, "uint8") if kind != "plain" else None
    o = O.decide_emit(rrs, rnd, budget, 0, dp, capacity=cap, scatter_index=sidx, shift_n=MAXQ)
    for _ in range(2):
        net.decideEmit(d_rrs[off:], d_rnd[off:], n, budget, 0, dp, d_norm[off:],
                       d_split[off:] if d_split is not None else None, d_queue, cap, d_size,
                       scatter_index=d_sidx, stream=stream())
        rc, flags = net.device_status(stream())
        total = int(host(d_size, np.uint32)[0])
        assert total == o["total"]
        assert np.array_equal(host(d_queue, np.uint32)[:min(total, cap)], o["queue"])
        assert np.array_equal(host(d_norm)[off:off + n].view(np.uint32),
                              o["rrs_norm"].view(np.uint32))
        if d_split is not None:
            assert np.array_equal(host(d_split)[off:off + n], o["split"])
        assert bool(flags & nb.DEV_OVERFLOW) == (total > cap)
