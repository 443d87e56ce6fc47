"""FP32 inference on several streams of one context: calls that do not decide keep nothing in the
context, so they may overlap with each other, with a captured graph and with a step. Each overlapped
result against the same call alone, bit for bit."""
import numpy as np
import pytest

import nrrs_b200 as nb
from gpu_util import empty, random_params, soa, stream, torch_cuda, upload

pytestmark = pytest.mark.gpu
NETS = {"64x2": (64, 2), "128x3": (128, 3), "shipped": None}
# a partial wave of tiles each, and several waves
SIZES = [(9_000, 12_345), (70_001, 50_021)]


def make(net):
    kw = dict(precision=nb.PREC_FP32, log2_hashmap_size=15, max_queue=1 << 17, max_train=256)
    if NETS[net] is None:
        cfg = nb.reference_config(**kw)
    else:
        w, h = NETS[net]
        cfg = nb.default_config(statnet_width=w, statnet_hidden=h, rrsnet_width=w, rrsnet_hidden=h,
                                **kw)
    ctx = nb.NRRSNetwork(cfg)
    random_params(ctx, 8)
    return ctx


class Call:
    """One way of inferring n vertices on stream s, and its outputs."""

    def __init__(self, ctx, kind, n, seed):
        torch = torch_cuda()
        self.ctx, self.kind, self.n, self.d = ctx, kind, n, upload(nb.synth(seed, n))
        sout = 6 if ctx.config.network == nb.NET_REFERENCE else 3
        self.out = {"stats": empty(sout * n), "rrs": empty(n)}
        self.sum = torch.zeros(1, dtype=torch.int64, device="cuda")
        self.n_dev = torch.tensor([n], dtype=torch.int32, device="cuda")
        self.extra = [empty(n), empty(n, "uint8"), empty(3 * n + 64, "int32"), empty(1, "int32")]
        self.dp = nb.default_decide()

    def run(self, s):
        v, n, o = soa(self.d), self.n, self.out
        if self.kind == "infer":
            self.ctx.inference(v, n, self.dp, o["stats"], o["rrs"], s)
        elif self.kind == "dev":
            self.ctx.inferDev(v, self.n_dev, n, self.dp, o["stats"], o["rrs"], s)
        elif self.kind == "accumulate":
            self.ctx.inferAccumulate(v, n, self.dp, o["stats"], o["rrs"], self.sum, s)
        else:
            norm, split, queue, size = self.extra
            self.ctx.generateRRSNumber(v, self.d["rnd"], n, n, 0, self.dp, o["stats"], o["rrs"],
                                       norm, split, queue, 3 * n + 64, size, s)

    def take(self):
        torch_cuda().cuda.synchronize()
        r = {k: t.cpu().numpy().view(np.uint32).copy() for k, t in self.out.items()}
        for t in self.out.values():
            t.zero_()
        return r


@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("kinds", [("infer", "infer"), ("infer", "step"), ("dev", "step"),
                                   ("accumulate", "accumulate"), ("graph", "infer"),
                                   ("graph", "step")])
@pytest.mark.parametrize("sizes", SIZES)
def test_overlapping_calls(net, kinds, sizes):
    torch = torch_cuda()
    ctx = make(net)
    a = Call(ctx, kinds[0].replace("graph", "infer"), sizes[0], 21)
    b = Call(ctx, kinds[1], sizes[1], 22)
    want = []
    for c in (a, b):
        c.run(stream())
        want.append(c.take())
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    if kinds[0] == "graph":
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=sa):
            a.run(stream())
        a.take()
    torch.cuda.synchronize()
    for _ in range(10):
        for _ in range(3):
            with torch.cuda.stream(sa):
                g.replay() if kinds[0] == "graph" else a.run(sa.cuda_stream)
            b.run(sb.cuda_stream)
        for c, w in zip((a, b), want):
            got = c.take()
            for k in w:
                assert np.array_equal(got[k], w[k]), (c.kind, k)
    ctx.close()
