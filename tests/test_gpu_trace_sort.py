"""The sorted trace's counting sort: every ray order gives nrrs_trace's hits, whatever the scratch's
(4-byte) alignment and however the rays fill the bins."""
import numpy as np
import pytest

import nrrs_b200 as nb
from gpu_util import stream, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("kind,n", [("spread", 70001), ("one_bin", 65536), ("spread", 65537)])
def test_sorted_trace_equals_trace(off, kind, n):
    torch = torch_cuda()
    scene = nb.Scene(*nb.synth_scene(3, n_boxes=20, closed=True))
    rng = np.random.default_rng(n + off)
    o = rng.uniform(0.1, 0.9, (n, 3)) if kind == "spread" else np.full((n, 3), 0.5)
    d = rng.normal(size=(n, 3)) if kind == "spread" else np.abs(rng.normal(size=(n, 3))) + 0.1
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    dev = lambda a, t=np.float32: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()  # noqa: E731
    rays = {"origin": dev(o), "dir": dev(d), "thp": dev(np.ones((n, 3))), "pdf": dev(np.zeros(n)),
            "pixel": dev(np.zeros(n), np.int32), "node": dev(np.zeros(n), np.int32)}
    n_dev = dev([n], np.int32)
    words = nb.trace_scratch_bytes(n) // 4
    scratch = torch.full((words + 8,), -1, dtype=torch.int32, device="cuda")
    out = []
    for srt in (False, True):
        h = {"prim": torch.full((n,), -7, dtype=torch.int32, device="cuda"),
             **{k: torch.zeros(n, device="cuda") for k in "tuv"}}
        R, H = nb.soa(nb.RaySoA, rays), nb.soa(nb.HitSoA, h)
        if srt:
            nb.trace_sorted(scene, R, n_dev, n, H, scratch[off:].data_ptr(), stream())
        else:
            nb.trace(scene, R, n_dev, n, H, stream())
        torch.cuda.synchronize()
        out.append(h)
    for k in out[0]:
        assert torch.equal(out[0][k], out[1][k]), k
    assert torch.all(scratch[off + words:] == -1)
    scene.close()
