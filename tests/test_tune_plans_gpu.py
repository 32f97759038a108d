"""The autotuner on sets of which the literal filter covers a part: it chooses by
the scans that are run, and matches stay exact."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def text(n, seed, planted):
    r = np.random.default_rng(seed)
    d = np.frombuffer(b"abcdefghijklmnopqrstuvwxyz0123456789_=:.- \n", dtype=np.uint8)[r.integers(0, 43, n)].copy()
    for at in range(0, n - 64, 4000):
        t = planted[int(r.integers(0, len(planted)))]
        d[at:at + len(t)] = np.frombuffer(t, dtype=np.uint8)
    return d


@pytest.mark.parametrize("literals", [[], [b"gamma ray", b"zebra"]])
def test_tuned_mixed_set(literals):
    # 400 regexes with prefixes, in several groups at the smaller limits, one
    # without and one with assertions
    import warpstate_b200 as ws
    r = np.random.default_rng(1)
    words = ["".join(chr(97 + int(c)) for c in r.integers(0, 16, int(r.integers(4, 12)))) for _ in range(800)]
    rx = [f"{a}[0-9]{{1,4}}{b}".encode() for a, b in zip(words[::2], words[1::2])]
    rx += [rb"[0-9]{1,3}\.[0-9]{3}x", rb"\bfatal: [0-9]"]
    planted = [f"{a}42{b}".encode() for a, b in zip(words[::2], words[1::2])][:60] + literals + [b"12.345x", b" fatal: 1"]
    pats = [(1, p) for p in rx] + [(0, p) for p in literals]
    b = ws.PatternSet.builder()
    for k, p in pats:
        b = b.literal_bytes(p) if k == 0 else b.regex(p.decode())
    ps = b.build()
    d, corpus = text(1 << 20, 2, planted), text(1 << 18, 3, planted)
    exp = oracle.scan_patterns(pats, d)
    assert len(exp) > 100
    m = ws.GpuMatcher.with_config(ps, ws.AutoMatcherConfig())
    walked = ws.GpuMatcher.with_config(ps, ws.AutoMatcherConfig().proposer(ws.PROPOSER_NONE))
    rep, all_walked = m.tune(corpus, flags=1), walked.tune(corpus, flags=1)
    for mm in (m, walked):
        assert np.array_equal(mm.scan_array(d), exp)
        assert np.array_equal(ws.StreamPipeline(mm).scan_array(d, block=100_003), exp.astype(np.uint64))
    # at the smallest limit the scans of `m` walk one group, those of `walked` several
    assert rep["groups_tried"][16384] < 0.75 * all_walked["groups_tried"][16384], (rep, all_walked)
    # with all in one automaton, the faster of the two ways is taken
    assert min(rep["groups_tried"].values()) < 1.1 * min(all_walked["groups_tried"].values()), (rep, all_walked)
    # tuned again, and pinned
    m.tune(corpus, flags=1)
    assert np.array_equal(m.scan_array(d), exp)
    m.set_walk(0, ws.PROPOSER_NONE)
    assert np.array_equal(m.scan_array(d), exp)
