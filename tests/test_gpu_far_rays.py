"""Rays from far away: distant origins against brute force, and rays from an infinite origin, which
miss everything without a walk through the tree."""
import numpy as np
import pytest

import nrrs_b200 as nb
import oracle as O
from gpu_util import host, stream, torch_cuda

pytestmark = pytest.mark.gpu


class Rays:
    """Rays on the device, their hits, and the shadow rays along them."""

    def __init__(self, o, d):
        torch = torch_cuda()
        n = self.n = len(o)
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()   # noqa: E731
        zero = np.zeros(n, np.int32)
        self.host = {"origin": o, "dir": d, "thp": np.ones((n, 3), np.float32),
                     "pdf": np.zeros(n, np.float32), "pixel": zero.view(np.uint32), "node": zero}
        r = {k: dev(a.view(np.int32) if a.dtype == np.uint32 else a) for k, a in self.host.items()}
        self.hits = {"prim": dev(zero), **{k: torch.zeros(n, device="cuda") for k in "tuv"}}
        self.n_dev, self.keep = dev(np.array([n], np.int32)), r
        self.rays, self.out = nb.soa(nb.RaySoA, r), nb.soa(nb.HitSoA, self.hits)

    def trace(self, scene):
        nb.trace(scene, self.rays, self.n_dev, self.n, self.out, stream())

    def ms(self, scene):
        torch = torch_cuda()
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        best = float("inf")
        for _ in range(3):
            e0.record()
            self.trace(scene)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best


# The slab test's error is below 1.8e-7 |lo - o| + 6e-8 |lo|; the boxes' growth of 1e-5 of the scene's
# extent and of the coordinates covers it to 55 extents.
@pytest.mark.parametrize("boxes,closed", [(5, False), (60, False), (60, True)])
@pytest.mark.parametrize("extents", [5, 20, 50])
@pytest.mark.parametrize("shift", [0.0, 100.0])
def test_distant_origins(boxes, closed, extents, shift):
    args = list(nb.synth_scene(3, n_boxes=boxes, closed=closed))
    args[0] = (np.asarray(args[0], np.float32).reshape(-1, 3) + np.float32(shift)).astype(np.float32)
    gs, hs = nb.Scene(*args), O.HostScene(*args)
    v, idx = args[0].astype(np.float64), np.asarray(args[1]).reshape(-1, 3)
    lo, hi = v.min(0), v.max(0)
    rng, n = np.random.default_rng(extents + boxes), 4000
    w = rng.dirichlet(np.ones(3), n)
    w[::4, 0] = 0.0                                    # an edge, and near it a vertex
    w[1::8] = np.eye(3)[rng.integers(0, 3, len(w[1::8]))]
    aim = np.einsum("nk,nkc->nc", w / w.sum(1, keepdims=True), v[idx[rng.integers(0, len(idx), n)]])
    d = rng.normal(size=(n, 3))
    d[rng.random((n, 3)) < 0.1] *= 1e-3                # grazing
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (aim - d * extents * (hi - lo).max()).astype(np.float32)
    d = aim - o
    r = Rays(o, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    r.trace(gs)
    want = hs.trace(r.host)
    assert host(r.hits["prim"]).view(np.uint32).tobytes() == want["prim"].tobytes()
    for k in "tuv":
        assert host(r.hits[k]).tobytes() == want[k].tobytes(), k
    assert (want["prim"] != 0xffffffff).mean() > 0.5
    gs.close()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [1, -1])
def test_infinite_origins_miss_at_the_root(axis, sign):
    scene = nb.Scene(*nb.synth_scene(3, n_boxes=1000, closed=True))
    rng, n = np.random.default_rng(7), 64
    o = rng.uniform(0.2, 0.8, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[::5, axis] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    near, far = Rays(o, d), o.copy()
    far[:, axis] = sign * np.inf
    far = Rays(far, d)
    far.trace(scene)
    assert (host(far.hits["prim"]).view(np.uint32) == 0xffffffff).all()
    # a walk over the 12,000 leaves takes a hundred times as long as an ordinary ray
    assert far.ms(scene) < 2 * near.ms(scene)
    scene.close()
