"""Host results around the size up to which one block orders them, and at match
capacities below it."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _matcher(cap):
    import warpstate_b200 as ws
    b = ws.PatternSet.builder().literal("ab").literal("abc").regex("abc[0-9]")
    return ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(cap))


PATS = [(0, b"ab"), (0, b"abc"), (1, b"abc[0-9]")]


@pytest.mark.parametrize("n", [0, 1, 2, 3, 341, 342, 682, 683, 1024, 3000])
def test_scan_and_batch_result_sizes(n):
    # three matches per "abc1", all with the same start
    import warpstate_b200 as ws
    m = _matcher(1 << 16)
    d = np.frombuffer(b"abc1 " * n + b"...", dtype=np.uint8)
    exp = oracle.scan_patterns(PATS, d)
    assert len(exp) == 3 * n
    assert np.array_equal(m.scan_array(d), exp)
    items = np.full(max(n, 1), 5, dtype=np.uint64)
    d5 = np.frombuffer((b"abc1 " * max(n, 1)), dtype=np.uint8)
    got = ws.scan_batch_packed(m, d5, items, ids=np.arange(len(items), dtype=np.uint64)[::-1].copy())
    assert len(got) == 3 * len(items)
    keys = [tuple(r) for r in got[:, [0, 2, 1, 3]].tolist()]
    assert keys == sorted(keys) and all(r[1] == 0 for r in keys)
    sp = ws.StreamPipeline(m).scan_array(d, block=777)
    assert np.array_equal(sp, exp.astype(np.uint64))


@pytest.mark.parametrize("cap", [1, 2, 3, 10, 2047, 2048, 2049])
def test_capacity_below_the_block_limit(cap):
    import warpstate_b200 as ws
    m = _matcher(cap)
    for n in (cap // 3, cap // 3 + 1):
        d = b"abc1 " * n
        if 3 * n > cap:
            with pytest.raises(ws.MatchBufferOverflow) as e:
                m.scan_array(d)
            assert e.value.count == 3 * n and e.value.max == cap
        else:
            assert len(m.scan_array(d)) == 3 * n
