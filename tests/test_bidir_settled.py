"""The settled filter of lazy labels (run_bidir_cta in
ddp_gb300/csrc/engine_bidir.cuh), restated as the steps that threads of one
wave may interleave in any order: two forward entries of u, and a reverse
entry of v at the other end of the arc (u, v).  Whatever the order, one side
must offer the length over u's smaller label."""
import pytest

W, GR = 5, 3  # the arc's weight, v's reverse label


def _installer(mem, node, dirn, g, other, every):
    """Steps of one entry: compare-and-swap of the label, filter bit, then
    the walk over the arc (the other node's bit, and on a hit its label)."""
    old = mem["label"].get((dirn, node))
    if old is not None and old <= g:
        return
    mem["label"][dirn, node] = g
    yield
    if every or old is None:
        mem["bit"].add((dirn, node))
    yield
    if (1 - dirn, other) not in mem["bit"]:
        return
    yield
    mem["mu"] = min(mem["mu"], g + W + mem["label"][1 - dirn, other])


def _orders(counts):
    """Every interleaving of threads with these numbers of steps."""
    if not any(counts):
        yield []
    for i, c in enumerate(counts):
        if c:
            for rest in _orders([x - (j == i) for j, x in enumerate(counts)]):
                yield [i] + rest


def _missed(every, labels):
    missed = 0
    for order in _orders([4] * (len(labels) + 1)):
        mem = {"label": {}, "bit": set(), "mu": 1 << 30}
        threads = [_installer(mem, "u", 0, g, "v", every) for g in labels]
        threads.append(_installer(mem, "v", 1, GR, "u", every))
        for i in order:
            next(threads[i], None)
        missed += mem["mu"] != min(labels) + W + GR
    return missed


@pytest.mark.parametrize("labels", [[10], [10, 8], [8, 10], [9, 9]])
def test_every_install_sets_the_bit(labels):
    assert _missed(True, labels) == 0


def test_a_bit_of_the_first_install_alone_misses_offers():
    assert _missed(False, [10]) == 0
    assert _missed(False, [10, 8]) > 0
