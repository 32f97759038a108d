"""Sets of regexes with and without prefixes: the groups that walk have the whole
chip, whatever groups wait behind the prefix filter."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

COVERED = [rb"key=[0-9]{1,9}", rb"alpha[ :]{1,3}[a-f]{2,4}", rb"user_[a-z0-9_]{1,9}\."]
WALKED = rb"[0-9]{1,3}\.[0-9]{3}x"


@pytest.mark.parametrize("n,chunk", [(1 << 25, 512), ((1 << 25) + 12345, 512), (1 << 22, 256)])
def test_chunks_of_the_walking_group(n, chunk):
    import warpstate_b200 as ws

    def build(rx):
        b = ws.PatternSet.builder()
        for p in rx:
            b = b.regex(p.decode())
        return ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 20).walk_chunk(chunk))

    r = np.random.default_rng(3)
    d = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz0123456789_=:.- \n", dtype=np.uint8)[r.integers(0, 43, n)].copy()
    for at in range(0, n - 16, 40_000):
        t = [b"key=12345 ", b"alpha: fade", b"12.345x"][at // 40_000 % 3]
        d[at:at + len(t)] = np.frombuffer(t, dtype=np.uint8)
    alone, mixed = build([WALKED]), build(COVERED + [WALKED])
    alone.scan_array(d)
    pats = [(1, p) for p in COVERED + [WALKED]]
    assert np.array_equal(mixed.scan_array(d), oracle.scan_patterns(pats, d))
    assert mixed.info()["n_groups"] == 2 and alone.info()["n_groups"] == 1
    # (last_chunks counts the chunks of every group without assertions)
    assert mixed.info()["last_chunks"] == 2 * alone.info()["last_chunks"]
