"""The find_iter chain over long candidate lists: windows of candidates that
overlap or not, clusters that go on past a window, lists of one tile and of
several, against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _text(kind, count, r):
    if kind == "digits":    # runs of digits: each digit starts a candidate
        return b" ".join(bytes(r.integers(48, 58, int(r.integers(1, 40))).astype(np.uint8)) for _ in range(count // 16 + 1))
    if kind == "words":     # a match holds hundreds of candidate starts
        return b"".join(b"a" * int(r.integers(1, 700)) + b"x=" for _ in range(count // 300 + 1))
    if kind == "long":      # ends beyond the parallel walk's limit
        return b"".join(b"b" * int(r.integers(900, 2600)) + (b"y" if k % 3 else b" ") for k in range(count // 1500 + 1))
    return b"k7= " * count  # apart


@pytest.mark.parametrize("count", [200, 257, 4096, 4099, 40_000])
@pytest.mark.parametrize("kind,regex", [("digits", rb"[0-9]{3,5}"), ("digits", rb"[0-9][0-9]|[0-9]{4}7"),
                                        ("words", rb"a+x"), ("words", rb"aa?a?x|[a-c]{200}"), ("long", rb"b+y|b{3}"),
                                        ("apart", rb"[a-z]7=")])
def test_chain_over_long_lists(kind, regex, count):
    import warpstate_b200 as ws
    text = _text(kind, count, np.random.default_rng(count))
    pats = [(1, regex), (1, rb"[x-z][ =]"), (0, b"zzz")]
    b = ws.PatternSet.builder().regex(regex.decode()).regex("[x-z][ =]").literal_bytes(b"zzz")
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 18))
    d = np.frombuffer(text, dtype=np.uint8)
    exp = oracle.scan_patterns(pats, d)
    assert np.array_equal(m.scan_array(d), exp)
    assert np.array_equal(m.scan_array(d), exp)  # (again with the capacities grown)
