"""The FP32 path at the edges of its tiles (64 samples), encoding tiles (128), weight-gradient stages
(64 samples) and chunks (256), and of its inference passes (1,048,576 vertices)."""
import sys
from pathlib import Path

import numpy as np
import pytest

import gpu_util as U

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
nb = U.nb

NETS = {"64x2": (64, 2), "64x3": (64, 3), "128x3": (128, 3), "shipped": None}


def make(net, **kw):
    if NETS[net] is None:
        cfg = nb.reference_config(precision=nb.PREC_FP32, log2_hashmap_size=14, **kw)
    else:
        w, h = NETS[net]
        cfg = nb.default_config(precision=nb.PREC_FP32, log2_hashmap_size=14, statnet_width=w,
                                statnet_hidden=h, rrsnet_width=w, rrsnet_hidden=h, **kw)
    n = nb.NRRSNetwork(cfg)
    rng = np.random.default_rng(5)
    ntab, nst, nrr = n.param_layout()
    p = np.concatenate([rng.uniform(-0.5, 0.5, ntab),
                        rng.uniform(-0.2, 0.2, nst + nrr)]).astype(np.float32)
    n.set_params(p)
    return n, p


def grads(net, t, a, b):
    """StatNet-side (table and StatNet) and RRSNet gradients of samples a .. b-1."""
    d = U.upload({k: np.ascontiguousarray(v[a:b]) for k, v in t.items()})
    net.trainGrads(U.soa(d), d["target"], b - a, None, U.stream())
    U.torch_cuda().cuda.synchronize()
    g = net.get_grads().astype(np.float64)
    ntab, nst, _ = net.param_layout()
    return g[:ntab + nst], g[ntab + nst:]


# The StatNet loss is a mean over samples, so a batch's gradient is the mean of its parts' ones,
# weighted by their sizes. Every sample's forward is the same sequence of FMAs wherever it sits, so
# only the order of the sums differs: at most 2^-24 sqrt(n) per sum, 1e-5 with room for n <= 2,000.
@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("n,cut", [(2, 1), (64, 63), (65, 64), (129, 1), (257, 128), (515, 256),
                                   (1700, 700)])
def test_fp32_gradients_add_up(net, n, cut):
    ctx, _ = make(net, max_queue=256, max_train=2048)
    t = nb.synth(11, n)
    t["target"] = np.minimum(t["target"], 10.0).astype(np.float32)
    whole, _ = grads(ctx, t, 0, n)
    a, _ = grads(ctx, t, 0, cut)
    b, _ = grads(ctx, t, cut, n)
    want = (cut * a + (n - cut) * b) / n
    assert np.linalg.norm(whole - want) <= 1e-5 * np.linalg.norm(want)
    ctx.close()


# against the FP64 oracle: the bar of the other FP32 gradient tests
@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("n", [1, 65])
def test_fp32_gradients_oracle(net, n):
    ctx, p = make(net, max_queue=256, max_train=256)
    t = nb.synth(12, n)
    t["target"] = np.minimum(t["target"], 10.0).astype(np.float32)
    s, r = grads(ctx, t, 0, n)
    g, _ = O.train_grads(ctx.config, p, t, t["target"], "f64")
    ntab, nst, _ = ctx.param_layout()
    for got, want in ((s, g[:ntab + nst]), (r, g[ntab + nst:])):
        assert np.linalg.norm(got - want) <= 2e-4 * np.linalg.norm(want)
    ctx.close()


@pytest.mark.parametrize("net", ["64x2", "128x3", "shipped"])
def test_fp32_inference_passes(net):
    """A queue longer than one pass, in one segment: the same bits as its ends alone."""
    n, k = (1 << 20) + 70, 300
    ctx, _ = make(net, max_queue=1 << 21, max_train=256)
    v = nb.synth(13, n)
    sout = 6 if net == "shipped" else 3

    def run(a, b):
        d = U.upload({x: np.ascontiguousarray(y[a:b]) for x, y in v.items()})
        stats, rrs = U.empty(sout * (b - a)), U.empty(b - a)
        ctx.inference(U.soa(d), b - a, nb.default_decide(), stats, rrs, U.stream())
        U.torch_cuda().cuda.synchronize()
        return stats.cpu().numpy().reshape(-1, sout), rrs.cpu().numpy()

    s, r = run(0, n)
    for a, b in ((0, k), (n - k, n), ((1 << 20) - k, (1 << 20) + 1)):
        s2, r2 = run(a, b)
        assert np.array_equal(s[a:b], s2) and np.array_equal(r[a:b], r2)
    ctx.close()
