"""The compacting filter with its gram table in L2 (thousands of literals of seven
bytes and more beside literals of one or two) against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("short", [[b"q"], [b"zq", b"!"]])
@pytest.mark.parametrize("n", [1, 15, 511, 513, 70_001, (1 << 20) + 3])
def test_large_set_with_short_literals(n, short):
    import warpstate_b200 as ws
    r = np.random.default_rng(7)
    lits = list({bytes(r.integers(97, 123, int(r.integers(7, 20))).astype(np.uint8)) for _ in range(9000)})
    d = r.integers(97, 123, n).astype(np.uint8)
    for at in range(0, n - 24, 301):
        t = lits[int(r.integers(0, len(lits)))]
        d[at:at + len(t)] = np.frombuffer(t, dtype=np.uint8)
    if n > 24:
        d[-len(lits[0]):] = np.frombuffer(lits[0], dtype=np.uint8)  # a match at the input's end
    pats = [(0, x) for x in lits + short]
    b = ws.PatternSet.builder()
    for _, x in pats:
        b = b.literal_bytes(x)
    exp = oracle.scan_patterns(pats, d)
    assert np.array_equal(ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig()).scan_array(d), exp)
    assert n < 513 or len(exp) > 1
