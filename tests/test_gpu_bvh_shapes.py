"""Traversal at the edges of the tree: a root that is a leaf, one pair, coincident triangles (ties
go to the lower index), and a tree cut off at its depth limit whose last leaf holds many triangles.
Closest hits against brute force, bit for bit; shadow rays against the closest hits."""
import numpy as np
import pytest

import nrrs_b200 as nb
import oracle as O
from gpu_util import host, stream, torch_cuda

pytestmark = pytest.mark.gpu


def triangles(kind):
    one = np.array([[0.2, 0.2, 0.5], [0.8, 0.25, 0.55], [0.4, 0.9, 0.45]], np.float32)
    if kind == "one":
        return one[None]
    if kind == "two":
        return np.stack([one, one + np.float32([0, 0, 0.2])])
    if kind == "equal":
        return np.repeat(one[None], 300, 0)
    # each binned cut takes the largest triangle off; the rest are coincident and halve
    k = np.float32(0.03) ** np.arange(18, dtype=np.float32)
    return np.concatenate([one[None] * k[:, None, None], np.repeat(one[None] * k[-1], 1 << 15, 0)])


@pytest.mark.parametrize("kind", ["one", "two", "equal", "depth_limit"])
def test_hits_of_extreme_trees(kind):
    torch = torch_cuda()
    v = triangles(kind)
    nt = len(v)
    args = (v.reshape(-1, 3), np.arange(3 * nt, dtype=np.uint32).reshape(nt, 3),
            np.zeros(nt, np.uint32), np.array([[0.5, 0.5, 0.5, 0, 0, 0]], np.float32),
            np.ones(3, np.float32))
    gs, hs = nb.Scene(*args), O.HostScene(*args)
    nodes, _, depth = gs.info()
    assert nodes <= 2 * nt - 1 and (depth == 31) == (kind == "depth_limit")
    n = 600
    rng = np.random.default_rng(7)
    o = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    w = rng.dirichlet(np.ones(3), n).astype(np.float32)
    aim = np.einsum("nk,nkc->nc", w, v[rng.integers(0, min(nt, 40), n)])
    d = (aim - o).astype(np.float32)
    d[::3] = rng.normal(size=d[::3].shape)
    d[1::9, 0] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    dev = lambda a, t=np.float32: torch.from_numpy(np.ascontiguousarray(a, t)).cuda()  # noqa: E731
    zero = np.zeros(n, np.int32)
    r = {"origin": o, "dir": d, "thp": np.ones((n, 3), np.float32), "pdf": np.zeros(n, np.float32),
         "pixel": zero.view(np.uint32), "node": zero}
    rays = {k: dev(a, np.int32 if a.dtype != np.float32 else np.float32) for k, a in r.items()}
    h = {"prim": dev(zero, np.int32), **{k: torch.zeros(n, device="cuda") for k in "tuv"}}
    n_dev = dev([n], np.int32)
    nb.trace(gs, nb.soa(nb.RaySoA, rays), n_dev, n, nb.soa(nb.HitSoA, h), stream())
    want = hs.trace(r)
    assert host(h["prim"]).view(np.uint32).tobytes() == want["prim"].tobytes()
    for k in "tuv":
        assert host(h[k]).tobytes() == want[k].tobytes(), k
    hit = want["prim"] != 0xffffffff
    assert hit.mean() > 0.2

    tmax = np.where(np.arange(n) % 2, np.where(hit, want["t"], 1), 2.0).astype(np.float32)
    tmax[2::4] = np.inf
    sh = {"origin": rays["origin"], "dir": rays["dir"], "tmax": dev(tmax),
          "contrib": dev(np.ones((n, 3))), "pixel": dev(zero, np.int32), "node": dev(zero, np.int32)}
    film, out = torch.zeros(1, 9, dtype=torch.int64, device="cuda"), torch.zeros(n, 3, device="cuda")
    nb.trace_shadow(gs, nb.soa(nb.ShadowSoA, sh), n_dev, n, film, out, stream())
    shadowed = hit & (want["t"] < tmax)
    assert np.array_equal(host(out)[:, 0] == 0, shadowed)
    gs.close()
