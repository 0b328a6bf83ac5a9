"""Hubs in the bidirectional searches: rows around the lengths at which a
team hands a row on in segments (512 arcs; segments of 256, longer ones past
1,024 of them), forward and reverse, on every record layout, in batches, single
queries and served requests.  Costs against the oracle, every path valid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub_graph(d, L, wmax, seed):
    """A hub with L arcs out (node 0), one with L arcs in (node 1), L nodes
    between them, and two random arcs a node."""
    rng = np.random.default_rng(seed)
    n = L + 40
    mid = np.arange(2, 2 + L)
    src = np.concatenate([np.zeros(L, np.int64), mid, rng.integers(0, n, 2 * n)])
    dst = np.concatenate([mid, np.ones(L, np.int64), rng.integers(0, n, 2 * n)])
    keep = src != dst
    src, dst = src[keep], dst[keep]
    o = np.argsort(src, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    return d.CSR(n, off, dst[o].astype(np.int32), rng.integers(1, wmax + 1, len(src)).astype(np.uint32))


@pytest.mark.parametrize("wmax", [4, 1000])
@pytest.mark.parametrize("L", [255, 511, 512, 513, 1025, 5000, 262143, 262145])
def test_rows_in_segments(gpu, oracle, L, wmax):
    d, O = gpu, oracle
    g = _hub_graph(d, L, wmax, L + wmax)
    rng = np.random.default_rng(L)
    q = 64 if L < 100000 else 16
    S, T = (rng.integers(0, g.n, q).astype(np.int32) for _ in range(2))
    # from and to the hubs, and to the nodes at the ends of segments
    S[:6], T[:6] = [0, 0, 0, 5, 2 + L - 1, 0], [1, 2 + L - 1, 2 + min(L - 1, 256), 1, 1, 3]
    gs = g.with_sentinel()
    want, _, _, done = O.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, S, T, hkind=0, mode=O.HEAP_POSMAP, threads=4,
                                    budget_s=1e9)
    assert done == q

    def check(p, i):
        if want[i] != d.INF:
            ok, why = O.check_path(g.off, g.col, g.w, p, int(S[i]), int(T[i]), int(want[i]))
            assert ok, (i, why)

    for coords in (False, True):
        dg = d.DeviceGraph.from_csr(g)
        if coords:
            dg.set_coords(rng.integers(0, 1000, (g.n, 2)).astype(np.int32))
            dg.set_euclid(0)  # potentials of 0: consistent whatever the coordinates
        dg.build_landmarks(8, seed=1, bits=8)
        kinds = [(d.H_BIDIR, {}), (d.H_BIDIR, {"block": 32}), (d.H_LANDMARK, {})]
        kinds += [(d.H_BIDIR_EUCLID, {})] if coords else [(d.H_BIDIR, {"flags": d.OPT_HASH})]
        for kind, kw in kinds:
            eng = d.BatchEngine(dg, kind, **kw)
            cost, _ = eng.solve(S, T)
            assert np.array_equal(cost, want), (coords, kind, kw)
            for i in range(0, q, 5):
                check(eng.path(i), i)
            eng.close()
        for i in range(8):
            r = dg.solve(int(S[i]), int(T[i]))
            assert r.cost == want[i]
            check(r.path, i)
        dg.close()
    dg = d.DeviceGraph.from_csr(g)
    srv = d.Server(dg, d.H_BIDIR, max_requests=256)
    first = srv.submit(S, T)
    ids, cost, _, _ = srv.drain()
    assert np.array_equal(cost, want[ids - first])
    srv.close()
    dg.close()


@pytest.mark.parametrize("hubs,L", [(1, 256), (1, 257), (1, 16384), (1, 16385), (1, 70000), (3, 5000), (9, 20000),
                                    (40, 300), (200, 60), (33, 257)])
def test_rows_in_narrow_phases(gpu, oracle, hubs, L):
    """Hubs met by the whole-grid search while one CTA runs its phases:
    rows in segments (one a team: 64 or 128), lists that the segments make too
    long, phases too wide in arcs; then the same graph under update batches."""
    d, O = gpu, oracle
    rng = np.random.default_rng(hubs * 1000 + L)
    mid, tail = 3000, 60
    n = 1 + hubs + mid + tail
    h, m0, t0 = 1, 1 + hubs, 1 + hubs + mid
    src = np.concatenate([np.zeros(hubs), np.repeat(h + np.arange(hubs), L), m0 + np.arange(mid),
                          t0 + np.arange(tail - 1)]).astype(np.int64)
    dst = np.concatenate([h + np.arange(hubs), m0 + rng.integers(0, mid, hubs * L), t0 + rng.integers(0, 20, mid),
                          t0 + 1 + np.arange(tail - 1)]).astype(np.int64)
    o = np.argsort(src, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    g = d.CSR(n, off, dst[o].astype(np.int32), rng.integers(1, 60, len(src)).astype(np.uint32))
    gs, s = g.with_sentinel(), 0

    def want(t, off=gs.off[:-1], col=gs.col, w=gs.w):
        f, c, _, _, _ = O.astar(len(off), off, col, w, np.zeros(len(off), np.int32), s, t, mode=O.HEAP_POSMAP)
        return c if f else d.INF

    dg = d.DeviceGraph.from_csr(g)
    for t in (n - 1, t0 + 7, m0 + 5, h + hubs - 1):
        hz = d.Heuristic(dg, t, d.H_USER, user_h=np.zeros(n, np.int32))
        c = want(t)
        for kw in ({}, {"K": 600}, {"grid": 3, "delta": 1}, {"delta": 100000}):
            r = dg.solve(s, t, hz, **kw)
            assert r.cost == c, (t, kw)
            if c != d.INF:
                ok, why = O.check_path(g.off, g.col, g.w, r.path, s, t, c)
                assert ok, (t, kw, why)
        hz.close()
    dg.close()
    for hk in (d.H_ZERO, d.H_BFS_HOPS):
        dg = d.DeviceGraph.from_csr(g)
        dyn = d.DynamicSearch(dg, s, n - 1, hk)
        off, col, w = gs.off[:-1].copy(), gs.col.copy(), gs.w.copy()
        assert dyn.cost == want(n - 1)
        for k in range(3):
            # the best path's arcs go, some come at new weights
            p = dyn.path()
            u = np.concatenate([p[:1], rng.integers(h, h + hubs, 30)]).astype(np.int32)
            v = np.concatenate([p[1:2], m0 + rng.integers(0, mid, 30)]).astype(np.int32)
            f = np.concatenate([[2], np.ones(30)]).astype(np.int32)
            x = rng.integers(1, 90, 31).astype(np.uint32)
            got = dyn.update(f, u, v, x)
            off, col, w, _ = O.apply_batch(len(off), off, col, w, f, u, v, x)
            assert got == want(n - 1, off, col, w), (hk, k)
        dyn.close()
        dg.close()


def test_queues_grow_with_the_arcs(gpu, oracle):
    """Hubs whose rows name every node many times: a phase pushes more entries
    than eight times the nodes."""
    d, O = gpu, oracle
    rng = np.random.default_rng(12)
    n, k, L = 1500, 6, 60000
    h = np.arange(k)
    src = np.concatenate([np.repeat(h, L), rng.integers(0, n, 4 * n), rng.integers(0, n, k * L // 4)])
    dst = np.concatenate([rng.integers(0, n, k * L), rng.integers(0, n, 4 * n), np.repeat(h, L // 4)])
    o = np.argsort(src, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
    g = d.CSR(n, off, dst[o].astype(np.int32), rng.integers(1, 1000001, len(src)).astype(np.uint32))
    S, T = (rng.integers(0, n, 24).astype(np.int32) for _ in range(2))
    gs = g.with_sentinel()
    want, _, _, done = O.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, S, T, hkind=0, mode=O.HEAP_POSMAP, threads=4,
                                    budget_s=1e9)
    assert done == len(S)
    dg = d.DeviceGraph.from_csr(g)
    dg.build_landmarks(16, seed=3, bits=8)
    eng = d.BatchEngine(dg, d.H_LANDMARK)
    assert np.array_equal(eng.solve(S, T)[0], want)
    eng.close()
    for i in range(24):
        for kw in ({"grid": 7}, {"K": 700}, {"delta": 50}, {"delta": 1000000}):
            assert dg.solve(int(S[i]), int(T[i]), **kw).cost == want[i], kw
    dg.close()
    dg = d.DeviceGraph.from_csr(g)
    dyn = d.DynamicSearch(dg, int(S[0]), int(T[0]), d.H_BFS_HOPS)
    assert dyn.cost == want[0]
    dyn.close()
    dg.close()
