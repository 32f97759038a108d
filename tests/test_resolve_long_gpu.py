"""Sets whose regexes all have prefixes, with candidate lists around and above
what one block resolves alone, while the prefix filter holds and after it gave
up (the walk's candidates, whose ends are still to be found), against the
oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

RX = [rb"key=[0-9]+", rb"user_[a-z0-9_]{0,9}\.", rb"abcd|abcdef|abcdefg", rb"(?:abcd)+", rb"open=[x ]+;", rb"\bword\b"]
BOUNDED = [rb"key=[0-9]{1,9}", rb"user_[a-z0-9_]{0,9}\.", rb"abcd|abcdef|abcdefg", rb"word [0-9]{2}"]


def build(pats, **cfg):
    import warpstate_b200 as ws
    b = ws.PatternSet.builder()
    for p in pats:
        b = b.regex(p.decode())
    return ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 19))


def text(counts, gap, seed):
    """`counts` of the texts of each kind, shuffled, about `gap` bytes apart."""
    r = np.random.default_rng(seed)
    kinds = [b"key=%d " % 1234, b"user_ab1.", b"abcdefg,", b"abcdabcdabcd;", b"open=xx;", b" word 12 "]
    order = r.permutation(np.repeat(np.arange(len(counts)), counts))
    return b"".join(kinds[k] + b"-" * int(r.integers(gap, gap + 9)) for k in order)


TRIP = b"open=" + b"x" * 3000 + b"key=1 "  # a walk of more than 1 KiB without a match
DENSE = b"abcdabcd" * 3000                 # more prefixes than the survivor list holds


@pytest.mark.parametrize("trip", [b"", TRIP, DENSE])
@pytest.mark.parametrize("pats", [RX, BOUNDED])
@pytest.mark.parametrize("counts", [(5, 1, 0, 3, 0, 2), (1023, 1024, 1025, 0, 7, 0), (4095, 0, 4096, 0, 4097, 1),
                                    (0, 30_000, 0, 1025, 0, 0), (9000, 9000, 9000, 9000, 9000, 9000)])
def test_lists_shared_by_blocks(counts, pats, trip):
    d = np.frombuffer(text(counts, 70, sum(counts)) + trip + text((1, 1, 1, 1, 1, 1), 3, 1), dtype=np.uint8)
    exp = oracle.scan_patterns([(1, p) for p in pats], d)
    assert len(exp) >= min(sum(counts), 6)
    m = build(pats)
    assert np.array_equal(m.scan_array(d), exp)
    assert np.array_equal(m.scan_array(d), exp)  # (again with the capacities grown)


@pytest.mark.parametrize("trip", [b"", TRIP])
def test_shared_lists_in_streams_and_batches(trip):
    import warpstate_b200 as ws
    pats = [(1, p) for p in RX]
    d = np.frombuffer(text((6000, 2000, 1500, 5000, 100, 100), 70, 9) + trip, dtype=np.uint8)
    m = build(RX)
    whole = oracle.scan_patterns(pats, d).astype(np.uint64)
    assert np.array_equal(ws.StreamPipeline(m).scan_array(d, block=400_001), whole)
    lens = np.full(len(d) // 4000, 4000, dtype=np.uint64)
    items = [(4000 * k, 4000) for k in range(len(lens))]
    got = ws.scan_batch_packed(m, d[:4000 * len(lens)], lens)
    assert np.array_equal(got, oracle.batch_scan(pats, d, items))


def test_overlapping_ends_merge_across_tiles():
    # every byte of a run ends a match, so that the walk lists a start many times
    # over, in several tiles
    pats = [rb"abcd[a-z]{1,9}", rb"abcd[a-z]*q"]
    r = np.random.default_rng(4)
    d = np.frombuffer(b"".join(b"abcd" + bytes(r.integers(97, 123, int(r.integers(1, 90))).astype(np.uint8)) + b" "
                               for _ in range(20_000)) + DENSE, dtype=np.uint8)
    exp = oracle.scan_patterns([(1, p) for p in pats], d)
    assert len(exp) > 20_000
    assert np.array_equal(build(pats).scan_array(d), exp)


@pytest.mark.parametrize("walked", [[], [rb"[0-9]{1,3}px"]])
def test_candidates_of_prefixes_overflow_and_are_counted(walked):
    # ten candidate starts per match: more than the candidate buffer holds on the
    # first try, whose counts size the second
    unit = b"abcd" * 10 + b" 12px " + b"-" * 754
    d = np.frombuffer(unit * ((24 << 20) // len(unit)), dtype=np.uint8)
    pats = [rb"(?:abcd)+", rb"key=[0-9]"] + walked
    exp = oracle.scan_patterns([(1, p) for p in pats], d)
    import warpstate_b200 as ws
    b = ws.PatternSet.builder()
    for p in pats:
        b = b.regex(p.decode())
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(70_000))
    assert len(exp) == (1 + len(walked)) * (len(d) // len(unit))
    assert np.array_equal(m.scan_array(d), exp)
    assert np.array_equal(m.scan_array(d), exp)
