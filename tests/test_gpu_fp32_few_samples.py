"""An FP32 training step of few samples scatters in one launch whatever the table's size; more samples
go by groups of levels. The same gradients either way."""
import numpy as np
import pytest

import gpu_util as U

pytestmark = pytest.mark.gpu
nb = U.nb
FEW = 16384


def step(log2, a, b):
    """Launches and gradients of samples a .. b-1."""
    net = U.make_net(precision=nb.PREC_FP32, log2_hashmap_size=log2, max_queue=256, max_train=FEW + 1)
    U.random_params(net, 5)
    t = nb.synth(3, b)
    t["target"] = np.minimum(t["target"], 10.0).astype(np.float32)
    d = U.upload({k: np.ascontiguousarray(v[a:]) for k, v in t.items()})
    k = net.launch_count()
    net.trainGrads(U.soa(d), d["target"], b - a, None, U.stream())
    k = net.launch_count() - k
    g = net.get_grads().astype(np.float64)[:sum(net.param_layout()[:2])]
    net.close()
    return k, g


@pytest.mark.parametrize("n", [1, 64, FEW])
def test_one_scatter_launch(n):
    assert step(20, 0, n)[0] == step(14, 0, n)[0]


# the StatNet gradient of a batch is the mean of its parts' ones, weighted by their sizes; the order of
# the FP32 sums differs, 2^-24 sqrt(n) per sum
def test_groups_and_one_launch_agree():
    few, g = step(20, 0, FEW)
    _, last = step(20, FEW, FEW + 1)
    groups, whole = step(20, 0, FEW + 1)
    assert groups == few + 2              # 110 MB of gradients in groups of at most 40
    want = (FEW * g + last) / (FEW + 1)
    assert np.linalg.norm(whole - want) <= 1e-5 * np.linalg.norm(want)
