"""The kernels' size rules (ddp_gb300/csrc/rules.h), compiled for the host:
the same functions that the device code calls, over the values at which they
change."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ddp_gb300", "csrc")
SHIM = """
#include "rules.h"
extern "C" {
int local_handback(int m, int list_cap, int64_t cap_q) { return ddp::local_handback(m, list_cap, cap_q); }
int block_threads(int want, int top) { return ddp::block_threads(want, top); }
int64_t long_row_arcs(int64_t len) { return ddp::long_row_arcs(len); }
int skewed_rows(int64_t in_long, int64_t arcs) { return ddp::skewed_rows(in_long, arcs); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, so = d / "rules.cpp", d / "rules.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-shared", "-fPIC", "-I" + CSRC, "-o", str(so), str(src)],
                   check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("cap_q", [1, 16, 300, 1535, 1536, 1537, 1 << 33])
def test_local_lists_hand_back_what_the_queue_holds(rules, cap_q):
    """A list that one CTA kept in shared memory never goes back past the
    end of a near queue shorter than it."""
    f = lambda m: rules.local_handback(m, 1536, C.c_int64(cap_q))  # noqa: E731
    for m in (0, 1, 15, 16, 17, 299, 301, 512, 513, 1535, 1536, 1537, 100000):
        assert f(m) == min(m, 1536, cap_q)


@pytest.mark.parametrize("top", [512, 1024])
def test_blocks_are_whole_warps(rules, top):
    for want in (1, 16, 31, 32, 33, 48, 100, 511, 512, 513, 1023, 1025, (1 << 31) - 1):
        got = rules.block_threads(want, top)
        assert got % 32 == 0 and got >= min(want, top) and got <= min(want + 31, top)


@pytest.mark.parametrize("e", [1, 15, 16, 1000, 5_000_000_000])
def test_graphs_with_hubs(rules, e):
    long_arcs, skew = rules.long_row_arcs, rules.skewed_rows
    long_arcs.restype = C.c_int64
    assert [long_arcs(C.c_int64(x)) for x in (0, 256, 257, 1 << 40)] == [0, 0, 257, 1 << 40]
    f = lambda k: bool(skew(C.c_int64(k), C.c_int64(e)))  # noqa: E731
    assert not f(0) and f(e) and f(max(e // 16, 1)) and (e // 16 < 2 or not f(e // 16 - 1))
