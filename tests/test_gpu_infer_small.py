"""The short-queue inference kernel (32 vertices per CTA) against the tiled one, bit for bit: a
context whose launch shape the caller chose keeps to the tiled kernel at every size."""
import numpy as np
import pytest

import nrrs_b200 as nb
from gpu_util import empty, soa, stream, torch_cuda, upload

pytestmark = pytest.mark.gpu

# network, the longest queue of one wave (CTAs per SM x 148 SMs x 32 vertices, whole 128-vertex tiles)
NETS = {"64x2": (64, 2, 4 * 148 * 32), "64x3": (64, 3, 3 * 148 * 32), "128x3": (128, 3, 148 * 32),
        "shipped": (32, 3, 4 * 148 * 32)}


def make(net, prec):
    w, h, _ = NETS[net]
    kw = dict(precision=prec, log2_hashmap_size=15, max_queue=1 << 16, max_train=256)
    cfg = nb.reference_config(**kw) if net == "shipped" else nb.default_config(
        statnet_width=w, statnet_hidden=h, rrsnet_width=w, rrsnet_hidden=h, **kw)
    n = nb.NRRSNetwork(cfg)
    rng = np.random.default_rng(3)
    ntab, nst, nrr = n.param_layout()
    n.set_params(np.concatenate([rng.uniform(-0.5, 0.5, ntab),
                                 rng.uniform(-0.2, 0.2, nst + nrr)]).astype(np.float32))
    return n


def step(net, d, n, dp, n_dev=None):
    sout = 6 if net.config.network == nb.NET_REFERENCE else 3
    o = dict(st=empty(sout * n), rrs=empty(n), norm=empty(n), split=empty(n, "uint8"),
             q=empty(3 * n + 64, "int32"), sz=empty(1, "int32"))
    if n_dev is None:
        net.generateRRSNumber(soa(d), d["rnd"], n, n, 0, dp, o["st"], o["rrs"], o["norm"],
                              o["split"], o["q"], 3 * n + 64, o["sz"], stream())
    else:
        net.generateRRSNumberDev(soa(d), d["rnd"], n_dev, n, n, 0, dp, o["st"], o["rrs"],
                                 o["norm"], o["split"], o["q"], 3 * n + 64, o["sz"],
                                 stream=stream())
    assert net.device_status(stream()) == (nb.OK, 0)
    return o


def same(a, b):
    for k in a:
        assert torch_cuda().equal(a[k], b[k]), k


@pytest.mark.parametrize("net", list(NETS))
@pytest.mark.parametrize("prec", [nb.PREC_FP16, nb.PREC_BF16])
def test_short_queue_same_bits(net, prec):
    small, tiled = make(net, prec), make(net, prec)
    tiled.set_launch_shape(0, 1)
    wave = NETS[net][2]
    for n in (1, 31, 32, 33, 127, 129, 3071, wave, wave + 1):
        d = upload(nb.synth(n, n))
        for src in (nb.FACTOR_RRSNET, nb.FACTOR_ADRRS):
            dp = nb.default_decide(factor_source=src)
            a, b = step(small, d, n, dp), step(tiled, d, n, dp)
            same(a, b)
        ctas = (n + 127) // 128 * 4
        assert small.last_infer_grid() == (ctas if n <= wave else tiled.last_infer_grid())
    small.close()
    tiled.close()


def test_short_queue_device_sizes_and_segments():
    torch = torch_cuda()
    small, tiled = make("64x2", nb.PREC_FP16), make("64x2", nb.PREC_FP16)
    tiled.set_launch_shape(0, 1)
    dp = nb.default_decide()
    bound = 1000
    d = upload(nb.synth(7, bound))
    for n in (0, 1, 129, bound):
        n_dev = torch.tensor([n], dtype=torch.int32, device="cuda")
        same(step(small, d, bound, dp, n_dev), step(tiled, d, bound, dp, n_dev))
    # three segments, one empty, with gaps between them
    segs = [nb.Segment(5, 200, 200, 0, 0, 600), nb.Segment(300, 0, 0, 0, 600, 10),
            nb.Segment(333, 77, 77, 0, 700, 300)]
    outs = []
    for net in (small, tiled):
        o = dict(st=empty(3 * bound), rrs=empty(bound), norm=empty(bound),
                 split=empty(bound, "uint8"), q=empty(1000, "int32"), sz=empty(3, "int32"))
        net.generateRRSNumberBatched(soa(d), d["rnd"], segs, dp, o["st"], o["rrs"], o["norm"],
                                     o["split"], o["q"], o["sz"], stream())
        assert net.device_status(stream()) == (nb.OK, 0)
        outs.append(o)
    same(*outs)
    small.close()
    tiled.close()
