"""Batches on graphs with coordinates, claimed longest first: at the sizes
around the number of slots, where the launch shape changes and past the
largest ranked batch, every query is answered once and at its own place, also
with equal distances, equal ends and ends on the graph's last node."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [151, 152, 153, 228, 380, 381, 912, 913, 8192, 8193])
def test_ranked_batches(gpu, oracle, q):
    d, O = gpu, oracle
    n = 600
    g = d.gen_geometric(n, 6, 1 << 16, 100000, 31)
    dg = d.DeviceGraph.from_csr(g)
    rng = np.random.default_rng(q)
    pool = [(0, 0), (n - 1, 0), (0, n - 1), (n - 1, n - 1)] + [tuple(x) for x in rng.integers(0, n, (56, 2))]
    pick = rng.integers(0, len(pool), q)
    S = np.array([pool[i][0] for i in pick], np.int32)
    T = np.array([pool[i][1] for i in pick], np.int32)
    gs = g.with_sentinel()  # the oracle's last row
    want, _, _, done = O.astar_many(gs.n, gs.off[:-1], gs.col, gs.w, np.array([x for x, _ in pool], np.int32),
                                    np.array([x for _, x in pool], np.int32), hkind=0, mode=O.HEAP_POSMAP,
                                    threads=4, budget_s=1e9)
    assert done == len(pool)
    eng = d.BatchEngine(dg)
    cost, _ = eng.solve(S, T)
    assert np.array_equal(cost, want[pick])
    for i in list(range(0, q, max(1, q // 20))) + [q - 1]:
        if cost[i] != d.INF:
            ok, why = O.check_path(gs.off, gs.col, gs.w, eng.path(i), int(S[i]), int(T[i]), int(cost[i]))
            assert ok, why
    cost2, _ = eng.solve(T, S)  # the buffers again, other queries
    back = {}
    for i in range(q):
        back.setdefault((int(T[i]), int(S[i])), int(cost2[i]))
        assert back[(int(T[i]), int(S[i]))] == int(cost2[i])
    eng.close()


def test_ranked_batch_on_device_pointers(gpu):
    torch = pytest.importorskip("torch")
    d = gpu
    n, q = 4000, 700
    g = d.gen_geometric(n, 6, 1 << 18, 100000, 77)
    dg = d.DeviceGraph.from_csr(g)
    rng = np.random.default_rng(3)
    eng = d.BatchEngine(dg)
    dS, dT, dc = (torch.empty(q, dtype=torch.int32, device="cuda") for _ in range(3))
    for _ in range(3):  # the first call captures, the others replay with new queries
        S, T = (rng.integers(0, n, q).astype(np.int32) for _ in range(2))
        dS.copy_(torch.from_numpy(S))
        dT.copy_(torch.from_numpy(T))
        torch.cuda.synchronize()
        eng.solve_device(q, dS.data_ptr(), dT.data_ptr(), dc.data_ptr())
        eng.sync()
        got = dc.cpu().numpy()
        cost, _ = eng.solve(S, T)
        assert np.array_equal(cost, got)
    eng.close()
