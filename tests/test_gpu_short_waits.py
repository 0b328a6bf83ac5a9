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
    env = dict(os.environ, DDP_NVCC_EXTRA="-DDDP_SPIN_LIMIT=256u")
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
m = d.gen_maze(300, 300, 0.25, 5)
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
