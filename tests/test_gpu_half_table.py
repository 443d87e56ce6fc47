"""The FP16 table's layout: its rows sit behind a shift that puts the hashed levels on 32-byte
sectors. Shifts of every size (the dense levels' rows modulo 8) against the FP32 path and the FP64
oracle, before and after an Adam step has rewritten the table."""
import sys
from pathlib import Path

import numpy as np
import pytest

import gpu_util as U

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
nb = U.nb


# base resolution and log2 entries: dense rows 0, 1, 3, 5, 6 and 7 modulo 8, an all-hashed grid
# and an all-dense one
@pytest.mark.parametrize("base,log2", [(3, 10), (4, 11), (16, 12), (5, 13), (6, 14), (16, 19),
                                       (64, 16), (2, 24)])
@pytest.mark.parametrize("cells", [True, False])
def test_half_table_shift(base, log2, cells):
    n, nt = 515, 300
    scale = 1.0 if (base, log2) == (2, 24) else 1.5
    net = nb.NRRSNetwork(nb.default_config(precision=nb.PREC_FP16, base_resolution=base,
                                           log2_hashmap_size=log2, per_level_scale=scale,
                                           max_queue=1024, max_train=512, lr=1e-3))
    if cells:
        try:
            net.set_cell_image(True)
        except nb.NRRSError:
            pytest.skip("no dense level")
    elif net.cell_image():
        net.set_cell_image(False)
    rng = np.random.default_rng(base)
    ntab, nst, nrr = net.param_layout()
    p = np.concatenate([rng.uniform(-0.5, 0.5, ntab),
                        rng.uniform(-0.15, 0.15, nst + nrr)]).astype(np.float32)
    net.set_params(p)
    dp = nb.default_decide()
    v, t = nb.synth(3, n), nb.synth(4, nt)
    for step in range(2):
        o = O.infer(net.config, net.get_params(), v, dp, "f64")
        stats, rrs = _infer(net, v, dp)
        # the mixed path's bars: factors 1e-2 relative, log-statistics 0.05
        assert np.max(np.abs(rrs - o["rrs"]) / o["rrs"]) < 1e-2
        assert np.max(np.abs(stats - o["stats"]) / np.maximum(1.0, np.abs(o["stats"]))) < 0.05
        if step == 0:
            _train(net, t, nt)
    net.close()


def _dev(a):
    import torch
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


def _soa(d):
    return nb.vertex_soa(d["pos"], d["wi"], d["normal"], d["roughness"], d["albedo"], d["thp"],
                         d["depth"], d["ref_mean"])


def _infer(net, v, dp):
    import torch
    n = len(v["rnd"])
    d = {k: _dev(a) for k, a in v.items()}
    stats = torch.zeros(n, 3, device="cuda")
    rrs = torch.zeros(n, device="cuda")
    net.inference(_soa(d), n, dp, stats, rrs, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return stats.cpu().numpy(), rrs.cpu().numpy()


def _train(net, t, n):
    import torch
    d = {k: _dev(a) for k, a in t.items()}
    net.train(_soa(d), d["target"], n, None, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
