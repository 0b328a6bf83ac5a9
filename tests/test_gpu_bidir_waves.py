"""The bidirectional wave search where its sizes change: bucket lists and
waves past their room, keys past the window, batch sizes at which a launch
takes another block size, small queues, and a search that floods its graph.
Costs against the oracle, every path valid."""
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


def _check(O, be, g, S, T, want):
    cost, plen = be.solve(S, T)
    assert np.array_equal(cost, want), np.flatnonzero(cost != want)[:8]
    for i in range(0, len(S), max(1, len(S) // 40)):
        p = be.path(i)
        assert len(p) == plen[i]
        if want[i] == INF:
            assert len(p) == 0
        else:
            ok, why = O.check_path(g.off, g.col, g.w, p, int(S[i]), int(T[i]), int(cost[i]))
            assert ok, (i, why)


def _fan(d, width, wlo, whi, seed):
    """s -> `width` nodes -> `width` nodes -> t, then back arcs to s."""
    rng = np.random.default_rng(seed)
    n = 2 * width + 2
    s, t = 0, n - 1
    A, Bn = np.arange(1, width + 1), np.arange(width + 1, 2 * width + 1)
    u = np.concatenate([np.full(width, s), np.repeat(A, 2), Bn, [t]])
    v = np.concatenate([A, rng.integers(width + 1, 2 * width + 1, 2 * width), np.full(width, t), [s]])
    w = rng.integers(wlo, whi + 1, len(u)).astype(np.uint32)
    o = np.argsort(u, kind="stable")
    off = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.int32)
    return d.CSR(n, off, v[o].astype(np.int32), w[o]), s, t


@pytest.mark.parametrize("width", [1, 31, 33, 1023, 1025, 4095, 4097, 20000])
@pytest.mark.parametrize("wlo,whi,delta", [(1, 1, 0), (0, 2, 0), (1, 1000, 1), (1, 1000, 5000), (5, 9, 3)])
def test_wide_buckets_and_windows(gpu, oracle, width, wlo, whi, delta):
    d = gpu
    g, s, t = _fan(d, width, wlo, whi, width + whi)
    dg = d.DeviceGraph.from_csr(g)
    rng = np.random.default_rng(width)
    S = np.concatenate([[s, t, s], rng.integers(0, g.n, 5)]).astype(np.int32)
    T = np.concatenate([[t, s, s], rng.integers(0, g.n, 5)]).astype(np.int32)
    want = _want(oracle, g, S, T)
    for kw in ({}, {"flags": d.OPT_HASH}, {"block": 64}, {"block": 1024}):
        be = d.BatchEngine(dg, d.H_BIDIR, delta=delta, grid=8, **kw)
        _check(oracle, be, g, S, T, want)
        be.close()
    # coordinates choose labels installed at once
    dg.set_coords(rng.integers(0, 1000, (g.n, 2)).astype(np.int32))
    be = d.BatchEngine(dg, d.H_BIDIR, delta=delta, grid=8)
    _check(oracle, be, g, S, T, want)
    be.close()
    dg.close()


@pytest.mark.parametrize("coords", [False, True])
def test_batch_sizes_and_small_queues(gpu, oracle, coords):
    d = gpu
    g = d.gen_random_chain(3000, 6, 1, 100, 17)
    dg = d.DeviceGraph.from_csr(g)
    rng = np.random.default_rng(3)
    if coords:
        dg.set_coords(rng.integers(0, 1000, (g.n, 2)).astype(np.int32))
    S = rng.integers(0, g.n, 1000).astype(np.int32)
    T = rng.integers(0, g.n, 1000).astype(np.int32)
    want = _want(oracle, g, S, T)
    be = d.BatchEngine(dg, d.H_BIDIR)
    for q in (1, 2, 152, 228, 229, 912, 913, 1000):
        _check(oracle, be, g, S[:q], T[:q], want[:q])
    be.close()
    # queues that some or all searches outgrow: re-run, exact
    for cap in (16, 256, 1024, 4096):
        be = d.BatchEngine(dg, d.H_BIDIR, grid=16, queue_cap=cap)
        _check(oracle, be, g, S[:40], T[:40], want[:40])
        be.close()
    dg.close()


def test_flooding_search_on_the_device_path(gpu, oracle):
    """Two parts of 60,000 nodes: a query across them explores one part from
    each end.  It outgrows the lazy form's memory and starts again."""
    torch = pytest.importorskip("torch")
    d = gpu
    a, b = d.gen_random_chain(60000, 12, 1, 100, 1), d.gen_random_chain(60000, 12, 1, 100, 2)
    g = d.CSR(a.n + b.n, np.concatenate([a.off[:-1], b.off + a.e]).astype(np.int32),
              np.concatenate([a.col, b.col + a.n]).astype(np.int32), np.concatenate([a.w, b.w]).astype(np.uint32))
    dg = d.DeviceGraph.from_csr(g)
    S = np.array([5, 60001, 7, 119999, 3], np.int32)
    T = np.array([90000, 9, 59999, 60000, 3], np.int32)
    want = _want(oracle, g, S, T)
    assert (want == INF).sum() == 2
    be = d.BatchEngine(dg, d.H_BIDIR, grid=2)
    dev = torch.device("cuda", 0)
    dS, dT = torch.from_numpy(S).to(dev), torch.from_numpy(T).to(dev)
    dc = torch.empty(len(S), dtype=torch.int32, device=dev)
    for _ in range(2):
        dc.fill_(-7)
        be.solve_device(len(S), dS.data_ptr(), dT.data_ptr(), dc.data_ptr(), 0)
        be.sync()
        assert np.array_equal(dc.cpu().numpy(), want)
    be.close()
    dg.close()


@pytest.mark.parametrize("wmin,wmax", [(0, 3), (1, 1), (1, 1000000)])
def test_hop_and_zero_bounds_agree_with_their_own_engine(gpu, oracle, wmin, wmax):
    """One-CTA slots answer these kinds bidirectionally; wider slots and
    DDP_OPT_SYNC run the A* engine.  Same costs, also on the layout that
    updates leave behind and for unreachable and equal endpoints."""
    d = gpu
    rng = np.random.default_rng(wmax)
    n, e = 3000, 9000  # no chain: some pairs are disconnected
    u = np.sort(rng.integers(0, n, e))
    off = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))]).astype(np.int32)
    g = d.CSR(n, off, rng.integers(0, n, e).astype(np.int32), rng.integers(wmin, wmax + 1, e).astype(np.uint32))
    dg = d.DeviceGraph.from_csr(g)
    S, T = rng.integers(0, n, 120).astype(np.int32), rng.integers(0, n, 120).astype(np.int32)
    T[:3] = S[:3]
    for rnd in range(2):
        want = _want(oracle, g, S, T)
        for kind in (d.H_ZERO, d.H_BFS_HOPS, d.H_BFS_CAPPED):
            for kw in ({}, {"flags": d.OPT_SYNC}, {"group": 2}, {"delta": 7}, {"queue_cap": 64}):
                be = d.BatchEngine(dg, kind, grid=12, **kw)
                _check(oracle, be, g, S, T, want)
                be.close()
        if rnd == 0:
            dj = rng.choice(e, 300, replace=False)
            dyn = d.DynamicSearch(dg, 0, 1, d.H_ZERO)
            iu, iv = rng.integers(0, n, 300).astype(np.int32), rng.integers(0, n, 300).astype(np.int32)
            dyn.update(np.concatenate([np.zeros(300, np.int32), np.ones(300, np.int32)]),
                       np.concatenate([u[dj], iu]), np.concatenate([g.col[dj], iv]),
                       np.concatenate([g.w[dj], rng.integers(wmin, wmax + 1, 300).astype(np.uint32)]))
            dyn.close()
            g = dg.read_csr()
    dg.close()
