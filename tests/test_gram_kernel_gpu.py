"""The gram kernel of the literal scan (one variant per shortest literal) at the
edges of its lanes, warp steps and inputs, bit-exact against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LETTERS = bytes(range(0x21, 0x7F))


def _set(shortest, count, alphabet, seed):
    r = np.random.default_rng(seed)
    al = np.frombuffer(alphabet, dtype=np.uint8)
    lits = {al[r.integers(0, al.size, shortest)].tobytes()}
    while len(lits) < count:
        lits.add(al[r.integers(0, al.size, int(r.integers(shortest, shortest + 12)))].tobytes())
    return sorted(lits)


# shortest literal -> grams: 3 bytes at every position, 4 bytes at every, every
# second, every fourth position, 16 bytes at every fourth (k-mers)
@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("shortest,count,alphabet",
                         [(3, 200, LETTERS), (4, 300, LETTERS), (5, 300, LETTERS), (6, 40, LETTERS), (7, 300, LETTERS),
                          (7, 12000, LETTERS), (19, 4000, b"ACGT")])
def test_gram_kernel_edges(shortest, count, alphabet, fold):
    import warpstate_b200 as ws
    lits = _set(shortest, count, alphabet, shortest)
    b = ws.PatternSet.builder().case_insensitive(fold)
    for p in lits:
        b = b.literal_bytes(p)
    m = ws.GpuMatcher.new(b.build())
    assert m.info()["filter_q"] == (3 if shortest == 3 else 16 if shortest == 19 else 4)
    pats = [(0, p) for p in lits]
    r = np.random.default_rng(11)
    al = np.frombuffer(alphabet, dtype=np.uint8)
    short = [p for p in lits if len(p) == shortest]
    for n in (1, 2, 3, 4, 15, 16, 17, 19, 31, 33, 63, 511, 512, 513, 527, 1023, 1024, 1025, 1031, 2048, 32768 + 5, 300_001):
        d = al[r.integers(0, al.size, n)].copy()
        # literals across lane, half-step and step boundaries, at the start and at the very end
        at = [0, 1, 2, 3, 13, 29, 500, 509, 511, 1009, 1021, 1023, 2045, 32765] + [int(x) for x in r.integers(0, n, 40)]
        for k, p in enumerate(at):
            lit = lits[int(r.integers(0, len(lits)))] if k % 3 else short[k % len(short)]
            if p + len(lit) <= n:
                d[p:p + len(lit)] = np.frombuffer(lit, dtype=np.uint8)
        tail = short[n % len(short)]
        if len(tail) <= n:
            d[n - len(tail):] = np.frombuffer(tail, dtype=np.uint8)
        got = m.scan_array(d)
        exp = oracle.scan_patterns(pats, d, case_insensitive=True) if fold else oracle.scan_patterns(pats, d)
        assert np.array_equal(got, exp), n
        if n >= shortest:
            assert len(exp) >= 1


def test_gram_kernel_list_overflow():
    # every position starts a literal: more survivors than the list holds, the
    # rest verified in place, with matches in the last bytes of the input
    import warpstate_b200 as ws
    for run in (b"zzz", b"zzzz", b"zzzzz", b"zzzzzzz"):
        lits = [run, run + b"z"] + _set(len(run), 300, LETTERS, 5)
        b = ws.PatternSet.builder()
        for p in lits:
            b = b.literal_bytes(p)
        m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(4 << 20))
        d = np.full((1 << 20) + 13, ord("z"), dtype=np.uint8)
        d[::4093] = ord("~")
        exp = oracle.scan_patterns([(0, p) for p in lits], d)
        assert len(exp) > (1 << 20)
        assert np.array_equal(m.scan_array(d), exp), run


@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("unit,n", [(b"zqz", 300_001), (b"zqzq", 262_144), (b"zqzqz", 300_013), (b"zqzqzqz", 524_303),
                                    (b"ACGTACGGTACCATGCATG", 400_007)])
def test_gram_kernel_full_list_forms(unit, n, fold):
    # the second look at every gram: each gram form, short and long literals,
    # runs of matches with gaps, both cases of a caseless set, an odd tail
    import warpstate_b200 as ws
    lits = sorted({unit, unit + unit[:2], unit + unit} | set(_set(len(unit), 200, LETTERS, 7)))
    b = ws.PatternSet.builder().case_insensitive(fold)
    for p in lits:
        b = b.literal_bytes(p)
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 20))
    period = len(unit) if len(unit) > 7 else 2
    d = np.frombuffer((unit[:period] * (n // period + 1))[:n], dtype=np.uint8).copy()
    d[np.random.default_rng(3).integers(0, n, n // 200)] = ord("~")
    if fold:
        d[::3] = np.frombuffer(d[::3].tobytes().swapcase(), dtype=np.uint8)
    pats = [(0, p) for p in lits]
    exp = oracle.scan_patterns(pats, d, case_insensitive=True) if fold else oracle.scan_patterns(pats, d)
    assert len(exp) > n // 32
    assert np.array_equal(m.scan_array(d), exp)
