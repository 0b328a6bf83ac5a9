"""Paths of the bidirectional searches on graphs with cycles of weight 0: the
forward and the reverse half may meet over such a cycle, and the path joined
from them must still visit no node twice (a path has at most n nodes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(d, n, seed, weights):
    rng = np.random.default_rng(seed)
    deg = rng.integers(1, 6, n)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    src = np.repeat(np.arange(n), deg)
    # half of the arcs to near nodes, some back: short cycles
    col = np.where(rng.random(off[-1]) < 0.6, (src + rng.integers(-3, 4, off[-1])) % n, rng.integers(0, n, off[-1]))
    w = rng.choice(np.array(weights, np.uint32), off[-1])
    return d.CSR(n, off, col.astype(np.int32), w)


def _check(O, g, p, s, t, cost):
    assert len(np.unique(p)) == len(p), ("a node twice", p)
    ok, why = O.check_path(g.off, g.col, g.w, p, s, t, cost)
    assert ok, why


def _wants(O, g, S, T):
    gs = g.with_sentinel()
    want, _, _, done = O.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, S, T, hkind=0, mode=O.HEAP_POSMAP, threads=4,
                                    budget_s=1e9)
    assert done == len(S)
    return want


@pytest.mark.parametrize("weights", [(0, 5), (0, 0, 0, 5), (0, 0, 1, 7)])
@pytest.mark.parametrize("n", [5, 23, 60, 400])
def test_batch_paths_are_simple(gpu, oracle, n, weights):
    d, O = gpu, oracle
    for seed in range(4):
        g = _graph(d, n, 100 * n + seed, weights)
        rng = np.random.default_rng(seed)
        S, T = (rng.integers(0, n, 120).astype(np.int32) for _ in range(2))
        want = _wants(O, g, S, T)
        for coords in (False, True):
            dg = d.DeviceGraph.from_csr(g)
            if coords:
                dg.set_coords(rng.integers(0, 100, (n, 2)).astype(np.int32))
            dg.build_landmarks(8, seed=1, bits=16)
            for kind, kw in ((d.H_ZERO, {}), (d.H_BFS_HOPS, {}), (d.H_BIDIR, {}), (d.H_BIDIR, {"flags": d.OPT_HASH}),
                             (d.H_LANDMARK, {})):
                eng = d.BatchEngine(dg, kind, **kw)
                cost, plen = eng.solve(S, T)
                assert np.array_equal(cost, want)
                for i in np.flatnonzero(cost != d.INF):
                    p = eng.path(int(i))
                    assert len(p) == plen[i] <= n
                    _check(O, g, p, int(S[i]), int(T[i]), int(cost[i]))
                eng.close()
            dg.close()


@pytest.mark.parametrize("weights", [(0, 5), (0, 0, 0, 5), (0, 0, 1, 7)])
@pytest.mark.parametrize("n", [5, 23, 60, 400])
def test_single_query_paths_are_simple(gpu, oracle, n, weights):
    d, O = gpu, oracle
    for seed in range(2):
        g = _graph(d, n, 100 * n + seed, weights)
        rng = np.random.default_rng(seed)
        S, T = (rng.integers(0, n, 40).astype(np.int32) for _ in range(2))
        want = _wants(O, g, S, T)
        for coords in (False, True):
            dg = d.DeviceGraph.from_csr(g)
            if coords:
                dg.set_coords(rng.integers(0, 100, (n, 2)).astype(np.int32))
            for s, t, c in zip(S.tolist(), T.tolist(), want.tolist()):
                for kw in ({}, {"grid": 4}):
                    r = dg.solve(s, t, **kw)
                    assert r.cost == c
                    if c == d.INF:
                        assert len(r.path) == 0
                    else:
                        _check(O, g, r.path, s, t, c)
            dg.close()


def test_long_paths_read_back_whole(gpu, oracle):
    """Paths longer than a slot keeps (1,024 nodes) are found again when they
    are asked for; length and nodes are of one path, although ties leave many."""
    d, O = gpu, oracle
    rng = np.random.default_rng(9)
    n = 7000
    src = np.repeat(np.arange(n), 8)
    col = np.clip(src + rng.integers(-5, 6, 8 * n), 0, n - 1)
    off = np.arange(0, 8 * n + 1, 8).astype(np.int32)
    g = d.CSR(n, off, col.astype(np.int32), rng.integers(1, 4, 8 * n).astype(np.uint32))
    S, T = np.arange(0, 40, 2).astype(np.int32), np.arange(n - 40, n, 2).astype(np.int32)
    want = _wants(O, g, S, T)
    dg = d.DeviceGraph.from_csr(g)
    for kind, kw in ((d.H_BIDIR, {}), (d.H_BFS_HOPS, {}), (d.H_ZERO, {"flags": d.OPT_SYNC})):
        eng = d.BatchEngine(dg, kind, **kw)
        cost, plen = eng.solve(S, T)
        assert np.array_equal(cost, want) and plen.min() > 1024
        for i in range(len(S)):
            p = eng.path(i)
            _check(O, g, p, int(S[i]), int(T[i]), int(cost[i]))
            assert np.array_equal(p, eng.path(i))
        eng.close()
    dg.close()
