"""Bucket edges of the bidirectional engine (edge and bucket in
ddp_gb300/csrc/engine_bidir.cuh), restated: the products by 2^64 / (2^32 /
width) never exceed 64 bits, start at or below the smallest key of the
bucket, and reach it in a step or two, for every width and bucket number."""
import random

import pytest

NONE = 0xFFFFFFFF
EDGES = [0, 1, 2, 3, 5, 1 << 16, (1 << 31) - 1, 1 << 31, (1 << 31) + 1, NONE - 1, NONE]


def _edge(b, rec):
    mul = ((1 << 64) - 1) // rec
    k = b * (mul >> 32) + ((b * (mul & NONE)) >> 32)
    assert k < 1 << 64
    steps = 0
    while k < NONE and (k * rec) >> 32 < b:
        k += 1
        steps += 1
    return min(k, NONE), steps


@pytest.mark.parametrize("seed", range(4))
def test_edge_is_the_smallest_key_of_its_bucket(seed):
    rng = random.Random(seed)
    widths = EDGES + [rng.getrandbits(rng.randint(1, 32)) for _ in range(400)]
    for dk in widths:
        rec = NONE if dk <= 1 else (1 << 32) // dk
        top = (NONE * rec) >> 32  # the last bucket a key can have
        for b in EDGES + [top, max(top - 1, 0)] + [rng.getrandbits(rng.randint(1, 32)) for _ in range(20)]:
            k, steps = _edge(b, rec)
            assert k == min(-(-(b << 32) // rec), NONE) and steps <= 2
            if k < NONE:
                assert (k * rec) >> 32 >= b and (k == 0 or ((k - 1) * rec) >> 32 < b)
