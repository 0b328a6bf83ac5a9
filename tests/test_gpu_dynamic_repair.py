"""Update batches at the sizes where the repair changes hands: subtrees and
hop floods too wide for one CTA, batches on either side of its limits, and
costs that rise past, fall below and return through the threshold of the
open list's cold tier (or lose the target altogether).  After every batch
cost and path equal a from-scratch A* on the updated graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scratch(O, off, col, w, s, t):
    n = len(off)
    h = np.maximum(O.bfs_heuristic(n, off, col, w, t), 0)
    found, cost, _, _, _ = O.astar(n, off, col, w, h, s, t)
    return cost if found else 2147483647


def _batch(rows):
    a = np.array(rows, np.int64).reshape(-1, 4)
    return a[:, 0].astype(np.int32), a[:, 1].astype(np.int32), a[:, 2].astype(np.int32), a[:, 3].astype(np.uint32)


@pytest.mark.parametrize("heur", ["hops", "zero"])
@pytest.mark.parametrize("group", [0, 1, 8])
def test_repair_hands_over_and_cold_tier(gpu, oracle, heur, group):
    d, O = gpu, oracle
    base = d.gen_random_chain(30000, 6, 1, 1000, 911)
    g = base.with_sentinel()
    s, t = int(base.perm[0]), int(base.perm[-1])
    dg = d.DeviceGraph.from_csr(g)
    dyn = d.DynamicSearch(dg, s, t, d.H_BFS_HOPS if heur == "hops" else d.H_ZERO, group=group)
    off, col, w = g.off[:-1].copy(), g.col.copy(), g.w.copy()
    rng = np.random.default_rng(5)
    n = len(off)
    ends = lambda: np.concatenate([off[1:], [len(col)]])

    def row(x):
        return [(int(col[j]), int(w[j])) for j in range(off[x], ends()[x])]

    def apply(rows):
        nonlocal off, col, w
        b = _batch(rows)
        cost = dyn.update(*b)
        off, col, w, _ = O.apply_batch(n, off, col, w, *b)
        want = _scratch(O, off, col, w, s, t)
        assert cost == want
        if want != d.INF:
            full = np.concatenate([off, [len(col)]]).astype(np.int32)
            ok, why = O.check_path(full, col, w, dyn.path(), s, t, cost)
            assert ok, why
        return cost

    c0 = dyn.cost
    # the source's arcs get heavier, and light again: nearly every label goes
    first = row(s)
    up = apply([(2, s, v, x + 700) for v, x in first])
    assert up >= c0 and dyn.stats()["invalidated"] > 1024
    assert apply([(2, s, v, x) for v, x in first]) == c0
    # the cost rises by cuts on the path, batch after batch
    for _ in range(4):
        p = dyn.path()
        assert apply([(0, int(p[i]), int(p[i + 1]), 0) for i in range(0, len(p) - 1, 3)]) >= c0
    # a hub next to the target: hops fall over most of the graph
    hub = int(base.perm[15000])
    apply([(1, hub, t, 900)] + [(1, int(x), hub, 950) for x in rng.integers(0, n, 300)])
    # shortcut: the cost falls; taking it out: it rises again
    low = apply([(1, s, t, 5)])
    assert low == 5
    assert apply([(0, s, t, 0)]) > low
    # batches of unrelated changes on both sides of one CTA's limit
    for m in (1, 2047, 2048, 2049, 4095, 4096, 4097):
        k = m // 2
        ins = [(1, int(a), int(b), int(x)) for a, b, x in zip(rng.integers(0, n, m - k), rng.integers(0, n, m - k),
                                                              rng.integers(1, 1001, m - k))]
        live = rng.choice(len(col), k, replace=False)
        tail = np.searchsorted(off, live, side="right") - 1
        apply(ins + [(0, int(tail[i]), int(col[live[i]]), 0) for i in range(k)])
    # the target is cut off, and comes back
    into = [(0, int(np.searchsorted(off, j, side="right") - 1), t, 0) for j in np.flatnonzero(col == t)]
    assert apply(into) == d.INF
    assert apply([(1, int(base.perm[7]), t, 3)]) < d.INF
    for _ in range(3):
        apply([(1, int(rng.integers(n)), int(rng.integers(n)), int(rng.integers(1, 1001)))])
    dyn.close()


@pytest.mark.parametrize("length", [1, 2, 4096, 4097, 6000])
def test_dynamic_paths_around_the_host_buffer(gpu, length):
    """A chain: the path has exactly `length` nodes, before and after a batch
    that changes the weight of its first arc (or of one beside it)."""
    d = gpu
    n = 6001
    e = np.arange(n - 1, dtype=np.int32)
    g = d.CSR(n, np.concatenate([e, [n - 1, n - 1]]).astype(np.int32), e + 1, np.full(n - 1, 2, np.uint32))
    dg = d.DeviceGraph.from_csr(g)
    dyn = d.DynamicSearch(dg, 0, length - 1, d.H_ZERO)
    assert np.array_equal(dyn.path(), np.arange(length)) and dyn.cost == 2 * (length - 1)
    assert dyn.update(*_batch([(2, 0, 1, 7)])) == (2 * (length - 1) + 5 if length > 1 else 0)
    assert np.array_equal(dyn.path(), np.arange(length))
    dyn.close()


def test_queues_grow_with_the_search(gpu, oracle):
    """Rows of hundreds of arcs push more entries than the queues are made
    for (twice the nodes): they grow, and every cost is exact."""
    d = gpu
    rng = np.random.default_rng(4)
    n, deg = 3000, 400
    off = np.arange(0, n * deg + 1, deg).astype(np.int32)
    col = rng.integers(0, n, n * deg).astype(np.int32)
    w = rng.integers(1, 1001, n * deg).astype(np.uint32)
    g = d.CSR(n, off, col, w)
    for hk in (d.H_BFS_HOPS, d.H_ZERO):
        dg = d.DeviceGraph.from_csr(g)
        dyn = d.DynamicSearch(dg, 5, 77, hk)
        o, c, ww = off[:-1].copy(), col.copy(), w.copy()

        def want():
            f, x, _, _, _ = oracle.astar(n, o, c, ww, np.zeros(n, np.int32), 5, 77, mode=oracle.HEAP_POSMAP)
            return x if f else d.INF
        assert dyn.cost == want()
        for k in range(4):
            p = dyn.path()
            # the path's arcs go, 300 others change
            j = rng.choice(n * deg, 300, replace=False)
            u = np.concatenate([p[:-1], j // deg]).astype(np.int32)
            v = np.concatenate([p[1:], col[j]]).astype(np.int32)
            f = np.concatenate([np.zeros(len(p) - 1, np.int32), np.full(300, 2, np.int32)])
            x = rng.integers(1, 1001, len(u)).astype(np.uint32)
            got = dyn.update(f, u, v, x)
            o, c, ww, _ = oracle.apply_batch(n, o, c, ww, f, u, v, x)
            assert got == want(), (hk, k)
        dyn.close()
        dg.close()


@pytest.mark.parametrize("kw", [{}, {"group": 1}, {"grid": 5}, {"K": 100}])
@pytest.mark.parametrize("extra", [0, 6000])
def test_targets_that_come_within_reach(gpu, oracle, kw, extra):
    """The target cannot be reached, or only from part of the graph, when the
    search is made; inserts open ways over nodes that had no hop bound, in one
    batch or several, some through heads of earlier inserts.
    extra: further inserts, so that the batch takes the host's path."""
    d = gpu
    rng = np.random.default_rng(3 + extra)
    part = d.gen_random_chain(800, 2, 1, 30, 8)
    k, n = 4, 4 * part.n
    src = np.repeat(np.arange(part.n), np.diff(part.off))
    src, dst = (np.concatenate([x + i * part.n for i in range(k)]) for x in (src, part.col))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    g = d.CSR(n, off, dst.astype(np.int32), rng.integers(1, 31, len(src)).astype(np.uint32))
    s, t = 5, n - 9
    for hk in (d.H_BFS_HOPS, d.H_ZERO):
        dg = d.DeviceGraph.from_csr(g)
        dyn = d.DynamicSearch(dg, s, t, hk, **kw)
        o, c, w = g.with_sentinel().off[:-1].copy(), g.col.copy(), g.w.copy()
        assert dyn.cost == d.INF

        def step(f, u, v, ww):
            nonlocal o, c, w
            more = rng.integers(0, part.n, (2, extra))  # inside the first part
            f, u = np.concatenate([f, np.ones(extra)]), np.concatenate([u, more[0]])
            v, ww = np.concatenate([v, more[1]]), np.concatenate([ww, np.full(extra, 1000)])
            f, u, v, ww = f.astype(np.int32), u.astype(np.int32), v.astype(np.int32), ww.astype(np.uint32)
            got = dyn.update(f, u, v, ww)
            o, c, w, _ = oracle.apply_batch(len(o), o, c, w, f, u, v, ww)
            f_, want, _, _, _ = oracle.astar(len(o), o, c, w, np.zeros(len(o), np.int32), s, t,
                                             mode=oracle.HEAP_POSMAP)
            assert got == (want if f_ else d.INF), (hk, got, want)

        at = lambda i: int(rng.integers(0, part.n)) + i * part.n  # noqa: E731
        step([1], [at(0)], [at(1)], [3])           # heads in reach of s, still no way
        step([1, 1], [at(2), at(1)], [at(3), at(1)], [5, 2])
        step([1], [at(1)], [at(2)], [4])           # now there is one
        step([0, 1, 1], [at(0), at(0), at(1)], [at(0), at(3), at(3)], [0, 40, 9])
        for _ in range(3):
            j = rng.choice(np.flatnonzero(c >= 0), 60, replace=False)
            src_now = np.repeat(np.arange(len(o)), np.diff(np.append(o, len(c))))
            step(rng.choice([0, 2], 60), src_now[j], c[j], rng.integers(1, 31, 60))
            step(np.ones(8), rng.integers(0, n, 8), rng.integers(0, n, 8), rng.integers(1, 60, 8))
        dyn.close()
        dg.close()


def test_bounds_past_the_largest_cost(gpu, oracle):
    """Hops times the least weight beyond 2^31: such nodes count as out of
    reach until inserts shorten their hops or a light arc lowers the bounds."""
    d = gpu
    n = 3000
    off = np.concatenate([np.arange(n), [n - 1]]).astype(np.int32)
    g = d.CSR(n, off, np.arange(1, n, dtype=np.int32), np.full(n - 1, 2_000_000, np.uint32))
    for light in (2_000_000, 7):
        dg = d.DeviceGraph.from_csr(g)
        dyn = d.DynamicSearch(dg, 0, n - 1, d.H_BFS_HOPS)
        assert dyn.cost == d.INF
        o, c, w = g.with_sentinel().off[:-1].copy(), g.col.copy(), g.w.copy()
        for u, v, x in ((900, 2100, light), (10, 880, light), (2300, 2990, light), (0, 5, light)):
            f, u, v, x = (np.array([a]) for a in (1, u, v, x))
            got = dyn.update(f, u, v, x)
            o, c, w, _ = oracle.apply_batch(len(o), o, c, w, f, u, v, x)
            f_, want, _, _, _ = oracle.astar(len(o), o, c, w, np.zeros(len(o), np.int32), 0, n - 1,
                                             mode=oracle.HEAP_POSMAP)
            assert got == (want if f_ else d.INF), (light, u, got, want)
        dyn.close()
        dg.close()


@pytest.mark.parametrize("kw", [{}, {"group": 1}, {"grid": 5}])
def test_inserts_into_nodes_out_of_reach(gpu, oracle, kw):
    """An arc into a node that cannot reach the target, then a shorter way to
    that arc's tail, then an arc from the node to the target."""
    d = gpu
    # 0 -> 1 (100), 1 -> 2 (200); the target is 2, node 3 has no arc out, 4 .. 9 a chain after it
    off = np.array([0, 1, 2, 2, 3, 4, 5, 6, 7, 8, 8], np.int32)
    g = d.CSR(10, off, np.array([1, 2, 4, 5, 6, 7, 8, 9], np.int32), np.array([100, 200, 1, 1, 1, 1, 1, 1], np.uint32))
    for hk in (d.H_BFS_HOPS, d.H_ZERO):
        for steps in ([(1, 1, 3, 1), (2, 0, 1, 10), (1, 3, 2, 5)],
                      [(1, 1, 3, 1), (1, 0, 3, 90), (2, 0, 1, 10), (1, 9, 2, 5)],
                      [(1, 0, 3, 150), (2, 0, 3, 120), (1, 1, 3, 1), (2, 0, 1, 10), (1, 6, 2, 5), (0, 1, 3, 0)],
                      [(1, 1, 3, 1), (0, 1, 3, 0), (1, 1, 3, 4), (2, 0, 1, 10), (1, 3, 2, 5)]):
            dg = d.DeviceGraph.from_csr(g)
            dyn = d.DynamicSearch(dg, 0, 2, hk, **kw)
            o, c, w = g.with_sentinel().off[:-1].copy(), g.col.copy(), g.w.copy()
            for i, st in enumerate(steps):
                f, u, v, x = _batch([st])
                got = dyn.update(f, u, v, x)
                o, c, w, _ = oracle.apply_batch(len(o), o, c, w, f, u, v, x)
                assert got == _scratch(oracle, o, c, w, 0, 2), (hk, steps, i)
            dyn.close()
            dg.close()
