"""A relaxation that loses to another one of the same node pushes nothing.  In
a graph of layers with unit arcs every path to a node has the same length, so a
search pushes and expands each node at most once, whatever its order and its bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(d, width, depth, arcs, seed):
    """`depth` layers of `width` nodes, `arcs` random arcs a node into the next
    layer; a source before the first and a target after the last."""
    rng = np.random.default_rng(seed)
    n = width * depth + 2
    s, t = n - 2, n - 1
    u = np.repeat(np.arange(width * (depth - 1)), arcs)
    v = (u // width + 1) * width + rng.integers(0, width, len(u))
    src = np.concatenate([u, np.full(width, s), np.arange(width) + width * (depth - 1)])
    dst = np.concatenate([v, np.arange(width), np.full(width, t)])
    o = np.argsort(src, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    return d.CSR(n, off, dst[o].astype(np.int32), np.ones(len(src), np.uint32)), s, t, depth + 1


@pytest.mark.parametrize("hk", ["H_BFS_HOPS", "H_ZERO"])
@pytest.mark.parametrize("width,depth,arcs,kw", [
    (64, 400, 24, {"K": 64}), (100, 60, 40, {"K": 100}), (33, 300, 16, {"K": 32, "grid": 5}),
    (2000, 12, 32, {}), (700, 40, 20, {"delta": 500}), (1025, 20, 20, {"block": 64})])
def test_each_node_once(gpu, width, depth, arcs, kw, hk):
    d = gpu
    g, s, t, length = _layers(d, width, depth, arcs, width)
    dg = d.DeviceGraph.from_csr(g)
    h = dg.heuristic(t, getattr(d, hk))
    for _ in range(3):
        r = dg.solve(s, t, h, **kw)
        assert r.cost == length
        assert r.stats[0] <= g.n and r.stats[2] <= g.n, r.stats  # expanded, pushed
    h.close()
    for group in (2, 4):
        eng = d.BatchEngine(dg, getattr(d, hk), group=group, **{k: v for k, v in kw.items() if k != "grid"})
        cost, _ = eng.solve(np.full(9, s, np.int32), np.full(9, t, np.int32))
        assert np.all(cost == length)
        eng.close()
    dg.close()
