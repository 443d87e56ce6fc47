"""FP32 contexts on a device with little memory left: the scratch that only serves speed is done
without (a step's features; the training step's own rows for the lane gradients and its finer
weight-gradient chunks), and what the context computes stays."""
import numpy as np
import pytest

import nrrs_b200 as nb
from gpu_util import empty, random_params, soa, stream, torch_cuda, upload

pytestmark = pytest.mark.gpu
NETS = {"64x2": (64, 2), "128x3": (128, 3), "shipped": None}
N, MAXQ, MAXT = 5_003, 1 << 20, 1 << 18
MB = 1 << 20


def make(net):
    kw = dict(precision=nb.PREC_FP32, log2_hashmap_size=15, max_queue=MAXQ, max_train=MAXT)
    if NETS[net] is None:
        cfg = nb.reference_config(**kw)
    else:
        w, h = NETS[net]
        cfg = nb.default_config(statnet_width=w, statnet_hidden=h, rrsnet_width=w, rrsnet_hidden=h,
                                **kw)
    return nb.NRRSNetwork(cfg)


def free():
    torch_cuda().cuda.empty_cache()
    return torch_cuda().cuda.mem_get_info()[0]


def outputs(net, d, soa_d):
    torch = torch_cuda()
    random_params(net, 4)
    sout = 6 if net.config.network == nb.NET_REFERENCE else 3
    o = dict(stats=empty(sout * N), rrs=empty(N), norm=empty(N), split=empty(N, "uint8"),
             queue=empty(3 * N + 64, "int32"), size=empty(1, "int32"))
    k0 = net.launch_count()
    net.generateRRSNumber(soa_d, d["rnd"], N, N, 0, nb.default_decide(), o["stats"], o["rrs"],
                          o["norm"], o["split"], o["queue"], 3 * N + 64, o["size"], stream())
    launches = net.launch_count() - k0
    net.trainGrads(soa_d, d["target"], N, None, stream())
    torch.cuda.synchronize()
    return {k: t.cpu().numpy().copy() for k, t in o.items()}, net.get_grads().astype(np.float64), launches


@pytest.mark.parametrize("net", list(NETS))
def test_context_in_little_memory(net):
    torch = torch_cuda()
    t = nb.synth(31, N)
    t["target"] = np.minimum(t["target"], 10.0).astype(np.float32)
    d = upload(t)
    v = soa(d)
    outputs(make(net), d, v)   # every kernel is loaded from here on
    whole = make(net)
    want, grads, launches = outputs(whole, d, v)
    layout = whole.param_layout()
    whole.close()
    before = free()
    whole = make(net)
    need = before - free()
    whole.close()
    features = 128 * MB                       # 1,048,576 vertices x 32 lanes
    lanes = (16 if NETS[net] is None else 32) * 4 * MAXT
    # the room that is left: a little less than everything; then less than everything but the features
    for short, compact in ((32 * MB, False), (features + lanes // 2 + 4 * MB, True)):
        hog = torch.empty(free() - (need - short), dtype=torch.uint8, device="cuda")
        small = make(net)
        del hog
        used = before - free()
        assert need - features - lanes - 64 * MB < used < need - features + 4 * MB
        assert (used < need - features - lanes // 2) == compact
        got, g, few = outputs(small, d, v)
        small.close()
        assert few == launches - 1            # no encoding kernel
        for k in want:
            assert np.array_equal(got[k], want[k]), k
        # the same products in FP32 sums of another order: 2^-24 sqrt(n) per sum, as where the
        # gradients of a batch's parts are added
        for a, b in ((0, sum(layout[:2])), (sum(layout[:2]), sum(layout))):
            assert np.linalg.norm(g[a:b] - grads[a:b]) <= 1e-5 * np.linalg.norm(grads[a:b])
