"""Waits that run out.  A second build of the library whose device waits give
up early runs in a process of its own: a call that outlasts them reports it,
and what comes after on the same handles is exact."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import sys
import numpy as np
import ddp_gb300 as d
from oracle import oracle as O
assert d.__file__.startswith(sys.argv[1])

def cost(g, s, t):
    gs = g.with_sentinel()
    f, c, _, _, _ = O.astar(gs.n, gs.off[:-1], gs.col, gs.w, np.zeros(gs.n, np.int32), s, t, mode=O.HEAP_POSMAP)
    return c if f else d.INF
"""


@pytest.fixture(scope="module")
def short_waits(gpu, oracle, tmp_path_factory):
    """Runs a script against the build with short waits."""
    root = tmp_path_factory.mktemp("short")
    for f in ("ddp_gb300", "include", "oracle"):
        shutil.copytree(os.path.join(ROOT, f), root / f, ignore=shutil.ignore_patterns("_build", "*.so", "__pycache__"))
    env = dict(os.environ, DDP_NVCC_EXTRA="-DDDP_SPIN_LIMIT=512u -DDDP_DYN_LEVELS=16 "
                                                 "-DDDP_SVC_POLLS=64u -DDDP_SVC_WAIT_NS=2000000LL")
    env.pop("PYTHONPATH", None)
    subprocess.run([sys.executable, "-m", "ddp_gb300.build"], cwd=root, env=env, check=True)

    def run(body):
        p = root / "body.py"
        p.write_text(HEAD + body)
        subprocess.run([sys.executable, str(p), str(root)], cwd=root, env=dict(env, PYTHONPATH=str(root)), check=True,
                       timeout=120)
    return run


def test_a_query_after_a_timed_out_one_is_exact(short_waits):
    """The grid waits for the phases that CTA 0 runs alone (milliseconds on
    a maze) and gives up; later queries read the same node labels."""
    short_waits("""
m = d.gen_maze(500, 500, 0.25, 5)
dg = d.DeviceGraph.from_csr(m)
rng = np.random.default_rng(1)
S, T = rng.integers(0, m.n, 8), rng.integers(0, m.n, 8)
for s, t in zip(S.tolist(), T.tolist()):
    try:
        dg.solve(0, m.n - 1, grid=8)
        raise SystemExit("the wait did not run out")
    except d.DdpError as e:
        assert e.code == 6, e
    r = dg.solve(s, t, flags=d.OPT_ONE_CTA)
    want = cost(m, s, t)
    assert r.cost == want, (s, t, r.cost, want)
    if want != d.INF:
        ok, why = O.check_path(m.off, m.col, m.w, r.path, s, t, want)
        assert ok, why
dg.close()
""")


def test_updates_given_up_on_leave_the_server_exact(short_waits):
    """Searches hold a version buffer for longer than an update waits: the
    update fails, its maintenance job is taken back (the next one writes its
    lists over), the service CTA stays, and later updates go through."""
    short_waits("""
import time
g = d.gen_geometric(300_000, 6, 1 << 20, 1000, 17, 4)
dg = d.DeviceGraph.from_csr(g)
srv = d.Server(dg, d.H_BIDIR, max_requests=128, versions=2, grid=2)
rng = np.random.default_rng(3)
# long queries: from one corner region to the opposite one
key = g.xy.sum(axis=1)
order = np.argsort(key)
q = 60
S, T = order[rng.integers(0, 3000, q)], order[-1 - rng.integers(0, 3000, q)]
src = np.repeat(np.arange(g.n, dtype=np.int32), np.diff(g.off))
w, versions, failed, batches = g.w.copy(), [g.w.copy()], 0, []
for k in range(24):  # made before the requests, which then outlast them
    j = rng.choice(g.e, 20000 if k % 2 else 200, replace=False)
    batches.append((j, rng.integers(1, 2000, len(j)).astype(np.uint32)))
first = srv.submit(S.astype(np.int32), T.astype(np.int32))
for j, more in batches:
    w[j] = w[j] + more
    try:
        srv.update(np.full(len(j), 2, np.int32), src[j], g.col[j], w[j])
        versions.append(w.copy())
    except d.DdpError as e:
        assert e.code == 6, e
        failed += 1
ids, costs, _, ver = srv.drain()
assert failed > 0, "no update ran into the wait"
assert srv.stats()["version"] == len(versions) - 1 and len(ids) == q
for k in range(0, q, 3):
    i = int(ids[k]) - first
    gv = d.CSR(g.n, g.off, g.col, versions[int(ver[k])])
    assert costs[k] == cost(gv, int(S[i]), int(T[i])), (i, int(ver[k]))
# nothing runs: an update and its answers
j = rng.choice(g.e, 5000, replace=False)
w[j] = w[j] + 7
srv.update(np.full(len(j), 2, np.int32), src[j], g.col[j], w[j])
srv.submit(S[:3].astype(np.int32), T[:3].astype(np.int32))
ids, costs, _, _ = srv.drain()
gv = d.CSR(g.n, g.off, g.col, w)
for k in range(len(ids)):
    i = int(ids[k]) - first - q
    assert costs[k] == cost(gv, int(S[i]), int(T[i]))
srv.close()
""")


def test_repairs_of_many_levels_hand_back(short_waits):
    """Chains of 3,000 nodes: an insert lowers hop bounds along one, a delete
    cuts the other near its source.  CTA 0 walks a level a node; the grid
    waits for a few levels at a time.  (K = 100 keeps the searches on the
    grid, whose waits are short.)"""
    short_waits("""
N = 3000
# s = 0, t = 1; forward chain 2 .. N+1 from s; chain N+2 .. 2N+1 into t by way of two nodes
s, t, f0, r0, a, b = 0, 1, 2, N + 2, 2 * N + 2, 2 * N + 3
src = [s, s] + list(range(f0, f0 + N - 1)) + [r0, a, b] + list(range(r0 + 1, r0 + N)) + [f0 + N - 1]
dst = [t, f0] + list(range(f0 + 1, f0 + N)) + [a, b, t] + list(range(r0, r0 + N - 1)) + [t]
w = [2 * N + 50] + [1] * (len(src) - 1)
n = 2 * N + 4
src, dst, w = (np.array(x) for x in (src, dst, w))
o = np.argsort(src, kind="stable")
off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
g = d.CSR(n, off, dst[o].astype(np.int32), w[o].astype(np.uint32))
for hk in (d.H_BFS_HOPS, d.H_ZERO):
    dg = d.DeviceGraph.from_csr(g)
    dyn = d.DynamicSearch(dg, s, t, hk, K=100)
    assert dyn.cost == N + 1
    # hops of the second chain fall by two, node after node; nothing else changes
    assert dyn.update([1], [r0], [t], [1]) == N + 1
    assert dyn.update([1], [s], [r0 + N - 1], [2 * N]) == N + 1
    # cut at the second node: 2,999 nodes lose their label, level by level
    assert dyn.update([0], [f0], [f0 + 1], [0]) == 2 * N + 50
    # and come back through an arc to the third
    got = dyn.update([1], [s], [f0 + 2], [4])
    assert got == 4 + N - 2, got
    dyn.close()
    dg.close()
""")


def test_a_failed_update_does_not_spoil_later_ones(short_waits):
    """A chain that CTA 0 follows for milliseconds: the update that opens it
    fails.  Later updates never answer from the labels it left."""
    short_waits("""
N = 6000
s, t, f0 = 0, 1, 2
src = [s, s] + list(range(f0, f0 + N))
dst = [t, f0] + list(range(f0 + 1, f0 + N)) + [t]
w = [5] + [1] * (len(src) - 1)
n = N + 4
off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.int32)
g = d.CSR(n, off, np.array(dst, np.int32), np.array(w, np.uint32))
for hk in (d.H_ZERO, d.H_BFS_HOPS):
    dg = d.DeviceGraph.from_csr(g)
    dyn = d.DynamicSearch(dg, s, t, hk, delta=1)
    assert dyn.cost == 5
    try:
        dyn.update([0], [s], [t], [0])
        raise SystemExit("the wait did not run out")
    except d.DdpError as e:
        assert e.code == 6, e
    try:
        assert dyn.update([1], [n - 1], [n - 2], [1]) == N + 1  # far from every path
    except d.DdpError as e:
        assert e.code == 6, e
    assert dyn.update([1], [s], [t], [7]) == 7
    assert dyn.update([1], [f0], [t], [3]) == 4
    assert dyn.path().tolist() == [s, f0, t]
    dyn.close()
    dg.close()
""")


def test_batches_after_a_timed_out_one_are_exact(short_waits):
    """Slots of several CTAs whose waits run out: their queries are run again
    alone, or fail, and later batches of the engine are exact or fail too, never
    wrong by the labels that were left."""
    short_waits("""
m = d.gen_maze(500, 500, 0.25, 5)
dg = d.DeviceGraph.from_csr(m)
rng = np.random.default_rng(2)
near = lambda q: (lambda a: (a, np.minimum(a + rng.integers(0, 4, q), m.n - 1)))(rng.integers(0, m.n, q))
eng = d.BatchEngine(dg, d.H_MANHATTAN, group=4, grid=6)
timed_out = 0
for rep in range(6):
    # long queries first: CTA 0 of a slot runs their phases, the others wait
    if rep % 2 == 0:
        S, T = rng.integers(0, m.n // 20, 12), rng.integers(m.n - m.n // 20, m.n, 12)
    else:
        S, T = near(40)
    S, T = S.astype(np.int32), T.astype(np.int32)
    want = [cost(m, int(s), int(t)) for s, t in zip(S, T)]
    try:
        got = eng.solve(S, T)[0].tolist()
        assert got == want, (rep, got, want)
    except d.DdpError as e:
        assert e.code == 6, e
        timed_out += 1
assert timed_out > 0, "no wait ran out"
eng.close()
dg.close()
""")
