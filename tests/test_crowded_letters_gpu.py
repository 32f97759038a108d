"""Literal sets that crowd their alphabet, on inputs over the same letters, on both
sides of the limits between the filter kernels, against the oracle."""
import random

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LOWER = b"abcdefghijklmnopqrstuvwxyz"


@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("letters,n,shortest", [(8, 45, 8), (8, 60, 8), (8, 300, 8), (26, 9000, 8), (26, 3500, 5), (12, 400, 5),
                                                (26, 5500, 4), (26, 7000, 4), (26, 180, 3), (26, 250, 3)])
def test_crowded_sets(letters, n, shortest, fold):
    import warpstate_b200 as ws
    r = random.Random(n)
    lits = sorted({bytes(r.choices(LOWER[:letters], k=r.randint(shortest, 14))) for _ in range(n)})
    g = np.random.default_rng(n)
    d = np.frombuffer(LOWER, dtype=np.uint8)[g.integers(0, letters, (2 << 20) + 77)].copy()
    for at in range(0, len(d) - 16, 5003):
        t = lits[at % len(lits)]
        d[at:at + len(t)] = np.frombuffer(t, dtype=np.uint8)
    if fold:
        up = g.integers(0, len(d), len(d) // 3)
        d[up] &= 0xDF
    b = ws.PatternSet.builder().case_insensitive(fold)
    for x in lits:
        b = b.literal_bytes(x)
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 22))
    exp = oracle.scan_patterns([(0, x) for x in lits], d, case_insensitive=fold)
    assert len(exp) > 10
    assert np.array_equal(m.scan_array(d), exp)
