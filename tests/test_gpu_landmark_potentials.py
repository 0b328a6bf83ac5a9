"""Landmark batches search bidirectionally with the landmark bounds as average
potentials: costs against the oracle and the A* engine, for every row width
(whole and odd numbers of 16-byte words), scaled and unscaled tables, nodes
that landmarks do not relate, and endpoints that are not connected."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
INF = 2147483647


def _want(O, g, S, T):
    gs = g.with_sentinel()
    cost, _, _, done = O.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, S, T, hkind=0, mode=O.HEAP_POSMAP,
                                    threads=os.cpu_count() or 1, budget_s=1e9)
    assert done == len(S)
    return cost


@pytest.mark.parametrize("bits,counts", [(8, (8, 16, 24, 64, 128)), (16, (4, 8, 12, 64))])
@pytest.mark.parametrize("kind", ["unit", "scaled", "split", "geo"])
def test_costs_for_every_row_width(gpu, oracle, bits, counts, kind):
    d = gpu
    rng = np.random.default_rng(bits)
    if kind == "split":  # no chain: landmarks miss nodes, pairs are disconnected
        n, e = 2000, 5000
        u = np.sort(rng.integers(0, n, e))
        off = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.int32)
        g = d.CSR(n, off, rng.integers(0, n, e).astype(np.int32), rng.integers(0, 90, e).astype(np.uint32))
    elif kind == "geo":
        g = d.gen_geometric(3000, 5, 1 << 16, 1000, 3)
    else:
        g = d.gen_random_chain(2500, 4, 1, 3 if kind == "unit" else 60000, 5)
    dg = d.DeviceGraph.from_csr(g)
    S, T = rng.integers(0, g.n, 150).astype(np.int32), rng.integers(0, g.n, 150).astype(np.int32)
    T[:3] = S[:3]
    want = _want(oracle, g, S, T)
    for count in counts:
        dg.build_landmarks(count, seed=count, bits=bits)
        for kw in ({}, {"block": 64, "grid": 4}, {"group": 2}, {"delta": 1}, {"flags": d.OPT_SYNC}):
            be = d.BatchEngine(dg, d.H_LANDMARK, **kw)
            cost, plen = be.solve(S, T)
            assert np.array_equal(cost, want), (count, kw, np.flatnonzero(cost != want)[:5])
            for i in range(0, len(S), 7):
                p = be.path(i)
                assert len(p) == plen[i]
                if want[i] != INF:
                    ok, why = oracle.check_path(g.off, g.col, g.w, p, int(S[i]), int(T[i]), int(cost[i]))
                    assert ok, why
            be.close()
    dg.close()


@pytest.mark.parametrize("count,bits", [(8, 8), (24, 8), (16, 16)])
@pytest.mark.parametrize("ways", [0, 1])
def test_pairs_without_a_path(gpu, oracle, count, bits, ways):
    """Two halves with no arcs between them, or arcs one way only: a landmark
    on the right side proves that there is no path and nothing is expanded;
    every cost equals the oracle's, reachable pairs and equal ends among them."""
    d = gpu
    a = d.gen_random_chain(1500, 4, 1, 100, 5)
    n, rng = 2 * a.n, np.random.default_rng(count + ways)
    src = np.repeat(np.arange(a.n), np.diff(a.off))
    s2, d2 = np.concatenate([src, src + a.n]), np.concatenate([a.col, a.col + a.n])
    if ways:
        s2, d2 = np.concatenate([s2, rng.integers(0, a.n, 50)]), np.concatenate([d2, rng.integers(a.n, n, 50)])
    o = np.argsort(s2, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(s2, minlength=n))]).astype(np.int32)
    g = d.CSR(n, off, d2[o].astype(np.int32), rng.integers(1, 101, len(s2)).astype(np.uint32))
    S, T = (rng.integers(0, n, 200).astype(np.int32) for _ in range(2))
    T[:5] = S[:5]
    gs = g.with_sentinel()
    want, _, _, done = oracle.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, S, T, hkind=0, mode=oracle.HEAP_POSMAP,
                                         threads=4, budget_s=1e9)
    assert done == len(S)
    dg = d.DeviceGraph.from_csr(g)
    dg.build_landmarks(count, seed=2, bits=bits)
    eng = d.BatchEngine(dg, d.H_LANDMARK)
    for _ in range(2):
        cost, plen = eng.solve(S, T)
        assert np.array_equal(cost, want)
        none = cost == d.INF
        assert none.any() and not none.all() and (plen[none] == 0).all()
        assert (eng.stats()[0][none, 0] == 0).mean() > 0.9  # expanded: nothing
    for i in range(0, 200, 7):
        if cost[i] != d.INF:
            ok, why = oracle.check_path(g.off, g.col, g.w, eng.path(i), int(S[i]), int(T[i]), int(cost[i]))
            assert ok, why
    eng.close()
    dg.close()


@pytest.mark.parametrize("bits,count", [(8, 8), (16, 8)])
@pytest.mark.parametrize("wmax", [900_000, 2_500_000, 150_000_000])
def test_distances_past_the_tables(gpu, oracle, bits, count, wmax):
    """A long chain with shortcuts and heavy arcs: landmark distances reach
    and pass the largest cost (2^31), so that a table's unreachable marker no
    longer proves that there is no path."""
    d = gpu
    rng = np.random.default_rng(wmax)
    n = 3000
    s, t = np.arange(n - 1), np.arange(1, n)
    e = rng.integers(0, n, 300)
    s, t = np.concatenate([s, e]), np.concatenate([t, np.minimum(e + rng.integers(1, 50, 300), n - 1)])
    o = np.argsort(s, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(s, minlength=n))]).astype(np.int32)
    g = d.CSR(n, off, t[o].astype(np.int32), rng.integers(1, wmax + 1, len(s)).astype(np.uint32))
    S = rng.integers(0, n, 200).astype(np.int32)
    T = np.minimum(S + rng.integers(0, 60 if wmax > 10_000_000 else 3000, 200), n - 1).astype(np.int32)
    want = _want(oracle, g, S, T)
    assert (want != INF).any()
    dg = d.DeviceGraph.from_csr(g)
    dg.build_landmarks(count, seed=3, bits=bits)
    for kw in ({}, {"group": 2}, {"flags": d.OPT_SYNC}):
        be = d.BatchEngine(dg, d.H_LANDMARK, **kw)
        cost, _ = be.solve(S, T)
        assert np.array_equal(cost, want), (kw, np.flatnonzero(cost != want)[:5])
        be.close()
    for i in range(0, 200, 20):
        h = dg.heuristic(int(T[i]), d.H_LANDMARK)
        assert dg.solve(int(S[i]), int(T[i]), h).cost == want[i]
        h.close()
    dg.close()
