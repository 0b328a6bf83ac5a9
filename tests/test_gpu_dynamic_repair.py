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
