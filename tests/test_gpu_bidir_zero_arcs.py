"""Bidirectional batches over paired records on graphs full of ties and of
arcs of weight 0: costs equal the oracle's and every parent chain is a path
of that cost (a tie that replaced a parent over a zero arc could close a
cycle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", [(0, 1), (0, 0, 0, 1), (0, 1, 2, 1000000), (1, 1, 1, 2)])
@pytest.mark.parametrize("n,deg", [(64, 8), (3000, 6), (20000, 24)])
def test_ties_and_zero_arcs(gpu, oracle, weights, n, deg):
    d, O = gpu, oracle
    g = d.gen_geometric(n, deg, 1 << 16, 100000, n)
    rng = np.random.default_rng(len(weights) + n)
    g.w[:] = rng.choice(np.array(weights, np.uint32), g.e)
    dg = d.DeviceGraph.from_csr(g)
    q = 160
    S, T = (rng.integers(0, n, q).astype(np.int32) for _ in range(2))
    gs = g.with_sentinel()
    want, _, _, done = O.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, S, T, hkind=0, mode=O.HEAP_POSMAP, threads=4,
                                    budget_s=1e9)
    assert done == q
    eng = d.BatchEngine(dg)
    cost, _ = eng.solve(S, T)
    assert np.array_equal(cost, want)
    for i in range(q):
        if cost[i] != d.INF:
            p = eng.path(i)
            assert len(p) <= n
            if len(p):  # longer than the engine keeps: none is given
                ok, why = O.check_path(gs.off, gs.col, gs.w, p, int(S[i]), int(T[i]), int(cost[i]))
                assert ok, why
    eng.close()
