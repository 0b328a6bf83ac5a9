"""Single queries: the bidirectional first attempt and the A* engine agree
with the oracle where the rule between them changes (weight ratio, budget,
options), on both record layouts, after updates, with paths longer than the
result block, and for heuristic arrays that are used again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cost(O, g, s, t):
    gs = g.with_sentinel()
    f, c, _, _, _ = O.astar(gs.n, gs.off[:-1], gs.col, gs.w, np.zeros(gs.n, np.int32), s, t, mode=O.HEAP_POSMAP)
    return c if f else 2147483647


def _check(O, g, r, s, t, want):
    assert r.cost == want
    if want == 2147483647:
        assert len(r.path) == 0
    else:
        ok, why = O.check_path(g.off, g.col, g.w, r.path, s, t, want)
        assert ok, why


@pytest.mark.parametrize("wmin,wmax", [(0, 3), (0, 4), (1, 3), (1, 4), (5, 19), (5, 20), (1, 1000000)])
@pytest.mark.parametrize("coords", [False, True])
def test_rule_between_the_engines(gpu, oracle, wmin, wmax, coords):
    d = gpu
    g = d.gen_random_chain(4000, 5, wmin, wmax, 7)
    dg = d.DeviceGraph.from_csr(g)
    rng = np.random.default_rng(wmax)
    if coords:
        dg.set_coords(rng.integers(0, 500, (g.n, 2)).astype(np.int32))
    for k in range(6):
        s, t = (int(x) for x in rng.integers(0, g.n, 2))
        t = s if k == 0 else t
        want = _cost(oracle, g, s, t)
        for kind in (None, d.H_BFS_HOPS, d.H_BFS_CAPPED):
            h = dg.heuristic(t, kind) if kind else None
            for kw in ({}, {"K": 64}, {"grid": 8}, {"delta": 3}, {"flags": d.OPT_ONE_CTA}, {}):
                _check(oracle, g, dg.solve(s, t, h, **kw), s, t, want)
            if h:
                h.close()
    # the layout that updates leave
    dj = rng.choice(g.e, 200, replace=False)
    src = np.repeat(np.arange(g.n, dtype=np.int32), np.diff(g.off))
    dyn = d.DynamicSearch(dg, 0, 1, d.H_ZERO)
    dyn.update(np.full(200, 2, np.int32), src[dj], g.col[dj], rng.integers(wmin, wmax + 1, 200).astype(np.uint32))
    dyn.close()
    g2 = dg.read_csr()
    s, t = (int(x) for x in rng.integers(0, g.n, 2))
    _check(oracle, g2, dg.solve(s, t), s, t, _cost(oracle, g2, s, t))
    dg.close()


def test_long_chains_and_budgets(gpu, oracle):
    """Paths of 4,095 to 12,300 nodes (result block, shared buffers), and a
    grid whose middle lies past the bidirectional budget."""
    d = gpu
    for n in (4095, 4096, 4097, 8193, 12300):
        off = np.concatenate([np.arange(n), [n - 1]]).astype(np.int32)
        g = d.CSR(n, off, np.arange(1, n, dtype=np.int32), np.ones(n - 1, np.uint32))
        dg = d.DeviceGraph.from_csr(g)
        for kw in ({}, {"grid": 4}, {"flags": d.OPT_ONE_CTA}):
            r = dg.solve(0, n - 1, **kw)
            assert r.cost == n - 1 and np.array_equal(r.path, np.arange(n))
            assert dg.solve(n - 1, 0, **kw).cost == d.INF
        dg.close()
    wall = np.zeros(400 * 400, np.uint8)
    g = d.grid_from_walls(400, 400, wall)
    g.w[:] = np.random.default_rng(1).integers(1, 30, g.e)
    bare = d.CSR(g.n, g.off, g.col, g.w)
    dg = d.DeviceGraph.from_csr(bare)
    s, t = 0, g.n - 1
    _check(oracle, bare, dg.solve(s, t), s, t, _cost(oracle, bare, s, t))
    dg.close()


def test_heuristic_arrays_are_reused(gpu, oracle):
    """Freed heuristics leave their arrays to the next ones: values of one
    target never show up under another, of either kind."""
    d = gpu
    g = d.gen_random_chain(3000, 4, 1, 9, 3)
    dg = d.DeviceGraph.from_csr(g)
    rng = np.random.default_rng(2)
    for k in range(8):
        t = int(rng.integers(0, g.n))
        hs = [dg.heuristic(x, d.H_BFS_HOPS, want_values=True) for x in (t, (t + 5) % g.n, (t + 9) % g.n)]
        for x, h in zip((t, (t + 5) % g.n, (t + 9) % g.n), hs):
            assert np.array_equal(h.values, oracle.bfs_heuristic(g.n, g.off[:-1], g.col, g.w, x))
        s = int(rng.integers(0, g.n))
        user = d.Heuristic(dg, t, d.H_USER, user_h=np.maximum(hs[0].values, 0))
        want = _cost(oracle, g, s, t)
        assert dg.solve(s, t, user).cost == want and dg.solve(s, t, hs[0], grid=8).cost == want
        for h in hs + [user]:
            h.close()
    dg.close()


@pytest.mark.parametrize("block", [1, 16, 31, 33, 48, 100, 511, 2000])
def test_blocks_of_any_size(gpu, oracle, block):
    """opts.block is taken up to whole warps by every engine."""
    d = gpu
    g = d.gen_random_chain(6000, 6, 1, 30, 11)
    dg = d.DeviceGraph.from_csr(g)
    s, t = 17, 4321
    want = _cost(oracle, g, s, t)
    h = dg.heuristic(t, d.H_BFS_HOPS)
    for kw in ({}, {"grid": 3}, {"K": 64}, {"flags": d.OPT_ONE_CTA}):
        for hh in (None, h):
            _check(oracle, g, dg.solve(s, t, hh, block=block, **kw), s, t, want)
    h.close()
    dg.close()
