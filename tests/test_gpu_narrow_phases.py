"""Searches whose phases cross the sizes at which one CTA takes over from the
grid and hands back (256 entries in, 512 out, 1,536 held in shared memory):
costs against the oracle, every path valid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layers(d, width, layers, wmin, wmax, seed):
    """s -> a layer of `width` nodes -> ... -> t, two random arcs per node
    into the next layer, then a chain of 40 nodes behind t."""
    rng = np.random.default_rng(seed)
    n = 2 + width * layers + 40
    rows = [[] for _ in range(n)]
    first = lambda k: 1 + k * width  # noqa: E731
    t = 1 + width * layers
    rows[0] = list(range(first(0), first(0) + width))
    for k in range(layers):
        for i in range(width):
            u = first(k) + i
            rows[u] = [t] if k == layers - 1 else (first(k + 1) + rng.integers(0, width, 2)).tolist()
    for i in range(t, n - 1):
        rows[i] = [i + 1]
    off = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate([np.array(r, np.int32) for r in rows if r]).astype(np.int32)
    w = rng.integers(wmin, wmax + 1, len(col)).astype(np.uint32)
    return d.CSR(n, off, col, w), 0, t


@pytest.mark.parametrize("width", [1, 2, 255, 256, 257, 511, 512, 513, 1535, 1537, 4000])
@pytest.mark.parametrize("wmin,wmax", [(1, 1), (0, 2), (1, 50)])
def test_phase_widths_match_oracle(gpu, oracle, width, wmin, wmax):
    d = gpu
    g, s, t = _layers(d, width, 4, wmin, wmax, 7 * width + wmax)
    gs = g.with_sentinel()
    dg = d.DeviceGraph.from_csr(g)
    h = dg.heuristic(t, d.H_BFS_HOPS)
    for target, hh in ((t, h), (t, None), (g.n - 1, None)):
        f, want, _, _, _ = oracle.astar(gs.n, gs.off[:-1], gs.col, gs.w, np.zeros(gs.n, np.int32), s, target)
        assert f
        for kw in ({}, {"K": 600}, {"K": 100}, {"grid": 2}, {"delta": 1000}):
            r = dg.solve(s, target, hh, **kw)
            assert r.cost == want, (target, kw)
            ok, why = oracle.check_path(g.off, g.col, g.w, r.path, s, target, r.cost)
            assert ok, why
    # nothing is reachable backwards
    assert dg.solve(t, s).cost == d.INF
    h.close()
    dg.close()


@pytest.mark.parametrize("width", [3, 300, 2000])
def test_update_batches_over_layers(gpu, oracle, width):
    """The resumed (keep mode) search through the same phase sizes."""
    d = gpu
    g, s, t = _layers(d, width, 3, 1, 20, width)
    dg = d.DeviceGraph.from_csr(g)
    dyn = d.DynamicSearch(dg, s, t, d.H_BFS_HOPS)
    rng = np.random.default_rng(width)
    off, col, w = g.with_sentinel().off[:-1].copy(), g.col.copy(), g.w.copy()
    for _ in range(6):
        k = min(width, 40)
        u = rng.integers(0, g.n - 42, 2 * k).astype(np.int32)
        live = np.array([x for x in u if g.off[x + 1] > g.off[x]], np.int32)
        v = g.col[g.off[live]]
        fl = np.where(np.arange(len(live)) % 2 == 0, 2, 0).astype(np.int32)
        ww = rng.integers(1, 30, len(live)).astype(np.uint32)
        got = dyn.update(fl, live, v, ww)
        off, col, w, _ = oracle.apply_batch(len(off), off, col, w, fl, live, v, ww)
        f, want, _, _, _ = oracle.astar(len(off), off, col, w, np.zeros(len(off), np.int32), s, t)
        assert got == (want if f else d.INF)
    dyn.close()
    dg.close()


@pytest.mark.parametrize("queue_cap", [1, 16, 300, 520, 1400, 1600])
@pytest.mark.parametrize("width", [200, 600, 1450, 4000])
def test_short_queues_overflow_or_answer(gpu, oracle, queue_cap, width):
    """A near queue shorter than the lists that one CTA keeps: the call
    answers exactly or reports the overflow, and the handle stays usable."""
    d = gpu
    g, s, t = _layers(d, width, 3, 1, 50, width + queue_cap)
    dg = d.DeviceGraph.from_csr(g)
    gs = g.with_sentinel()
    f, want, _, _, _ = oracle.astar(gs.n, gs.off[:-1], gs.col, gs.w, np.zeros(gs.n, np.int32), s, t)
    for _ in range(2):
        try:
            assert dg.solve(s, t, queue_cap=queue_cap).cost == want
        except d.DdpError as e:
            assert e.code == 5
    assert dg.solve(s, t).cost == want
    dg.close()
