"""Which kernel a short queue of the tensor-core path takes: its own, unless the caller chose a launch
shape or an inference mode other than the default."""
import pytest

import nrrs_b200 as nb
from gpu_util import empty, make_net, random_params, soa, stream, torch_cuda, upload

pytestmark = pytest.mark.gpu
N = 3071


def test_route_follows_the_choice():
    net = make_net(precision=nb.PREC_FP16, max_queue=1 << 16, max_train=256)
    random_params(net, 6)
    d, dp, stats, rrs = upload(nb.synth(9, N)), nb.default_decide(), empty(3 * N), empty(N)
    out = []

    def short():
        net.inference(soa(d), N, dp, stats, rrs, stream())
        torch_cuda().cuda.synchronize()
        out.append((stats.cpu(), rrs.cpu()))
        return net.last_infer_grid() == (N + 127) // 128 * 4   # 32 vertices per CTA

    assert short()
    net.set_infer_split(0)            # the default
    assert short()
    net.set_infer_split(2)
    assert not short()
    net.set_infer_split(0)
    assert short()
    net.set_launch_shape(0, 1)
    assert not short()
    net.set_infer_split(0)            # takes back the mode, not the shape
    assert not short()
    net.autotune(1 << 15)
    assert short()
    for s, r in out[1:]:
        assert torch_cuda().equal(s, out[0][0]) and torch_cuda().equal(r, out[0][1])
    net.close()
