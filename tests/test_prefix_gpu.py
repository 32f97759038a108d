"""Regex candidates from the literal filter (regexes whose matches begin with
known prefixes) against the oracle and against the walk of the same set."""
import numpy as np
import pytest

import oracle
import workloads as w

pytestmark = pytest.mark.gpu

LOG = b"abcdefghijklmnopqrstuvwxyz0123456789_=:.- \n"


def build(pats, fold=False, **cfg):
    import warpstate_b200 as ws
    b = ws.PatternSet.builder().case_insensitive(fold)
    for k, p in pats:
        b = b.literal_bytes(p) if k == 0 else b.regex(p.decode())
    c = ws.AutoMatcherConfig()
    for k, v in cfg.items():
        getattr(c, k)(v)
    return ws.GpuMatcher.with_config(b.build(), c)


def text(n, seed, alphabet=LOG):
    r = np.random.default_rng(seed)
    return np.frombuffer(alphabet, dtype=np.uint8)[r.integers(0, len(alphabet), n)].copy()


def plant(d, texts, every, seed):
    r = np.random.default_rng(seed)
    for at in range(0, len(d) - 64, every):
        t = texts[int(r.integers(0, len(texts)))]
        o = at + int(r.integers(0, max(1, min(every, 64) - 1)))
        if o + len(t) <= len(d):
            d[o:o + len(t)] = np.frombuffer(t, dtype=np.uint8)
    return d


RX = [rb"key=[0-9]+", rb"(?:alpha|beta1|gamma)[ :]{1,3}[a-f]{2,4}", rb"user_[a-z0-9_]*\.", rb"abcd|abcdef|abcdefg",
      rb"(?:abcd)+", rb"\bfatal\b", rb"^stamp=[0-9]{2,4}", rb"done: ok$", rb"tail[a-z]{1,6}", rb"\Aabcd", rb"last0\z"]
TEXTS = [b"key=12345", b"alpha: fade", b"beta1 ab", b"user_a1_b.", b"abcdefg", b"abcdabcdabcd", b" fatal ", b"fatality",
         b"\nstamp=123", b"done: ok\n", b"done: okay", b"tailwind", b"user_no_end", b"key=", b"alpha;;"]


@pytest.mark.parametrize("extra", [[], [(0, b"gamma ray"), (0, b"abcd"), (0, b"xyz"), (1, rb"[a-c]{2}9[a-c]+")],
                                   [(0, b"q"), (0, b"key=1")]])
@pytest.mark.parametrize("n", [9, 64, 4096, 100_003, (1 << 20) + 5])
def test_prefix_candidates_vs_oracle_and_walk(extra, n):
    # literal-free, mixed with literals of 3 bytes and a regex that is walked,
    # and with a one-byte literal (the compacting filter)
    pats = [(1, p) for p in RX] + extra
    d = plant(text(n, n), TEXTS, 97 if n < 200_000 else 311, n)
    d[-9:] = np.frombuffer(b"abcdlast0", dtype=np.uint8)  # a match at the input's end
    exp = oracle.scan_patterns(pats, d)
    assert len(exp) >= 2
    assert np.array_equal(build(pats, max_matches=1 << 20).scan_array(d), exp)
    assert np.array_equal(build(pats, max_matches=1 << 20, proposer=1).scan_array(d), exp)


def test_prefix_filter_gives_up_and_walks():
    # the cases the filter leaves to the walk at run time: prefixes everywhere
    # (more survivors than the list holds), walks longer than 1 KiB without a
    # match, many long walks; and a set with one group of each kind
    long_open = b"open=" + b"x" * 5000 + b";"
    runs = (b"key=" + b"k" * 200 + b" ") * 3000
    dense = b"abcd" * 60_000
    pats = [(1, rb"open=[x ]+;"), (1, rb"key=k+;"), (1, rb"abcd[a-d]{1,6}"), (1, rb"\bword\b"), (1, rb"[a-c]{2}9[a-c]+"),
            (0, b"dabc")]
    base = plant(text(200_000, 3), [b"open=xx;", b"key=kkk;", b" word ", b"ab9c"], 500, 4).tobytes()
    for data in (base, base + long_open + base, base + runs + base, base + dense + base, b"open=" + b"x" * 3000):
        exp = oracle.scan_patterns(pats, data)
        got = build(pats, max_matches=1 << 20).scan_array(data)
        assert np.array_equal(got, exp), len(data)


def test_prefix_batch_stream_and_caseless():
    import warpstate_b200 as ws
    pats = [(1, p) for p in RX[:9]] + [(0, b"Gamma"), (0, b"abcd")]
    r = np.random.default_rng(5)
    lens = r.integers(1, 3000, size=300)
    total = int(lens.sum())
    ends = np.cumsum(lens)
    d = plant(text(total, 6), TEXTS, 150, 7)
    for e in ends[:-1]:  # prefixes and matches cut by item ends
        t = TEXTS[int(e) % len(TEXTS)]
        if e + 10 < total:
            d[e - 5:e - 5 + len(t)] = np.frombuffer(t, dtype=np.uint8)[:total - e + 5]
    items = [(int(e - n), int(n)) for e, n in zip(ends, lens)]
    m = build(pats, window_mib=1)
    got = ws.scan_batch_packed(m, d, lens.astype(np.uint64))
    exp = oracle.batch_scan(pats, d, items)
    assert len(exp) > 300 and np.array_equal(got, exp)
    big = np.concatenate([d] * 5)
    whole = oracle.scan_patterns(pats, big).astype(np.uint64)
    for block in (777, 65_537, 1 << 20):
        part = big if block > 777 else big[:60_000]
        ref = whole if block > 777 else oracle.scan_patterns(pats, part).astype(np.uint64)
        assert np.array_equal(ws.StreamPipeline(m).scan_array(part, block=block), ref), block
    folded = np.frombuffer(big.tobytes().replace(b"abcd", b"aBcD"), dtype=np.uint8)
    exp = oracle.scan_patterns(pats, folded, case_insensitive=True)
    assert np.array_equal(build(pats, fold=True).scan_array(folded), exp)


def test_prefix_nucleotides_long_grams():
    # degenerate motifs without k-mers: 16-byte grams of 20-byte prefixes
    rx = w.gen_iupac(60, 5 * 1000 + 2)
    r = w.Rng(77)
    d = w.fill_acgt(1 << 20, 5)
    texts = [bytes(r.choice(w.IUPAC.get(c, c)).encode()[0] for c in pos) for _, pos in rx]
    d = plant(d, texts, 4096, 8)
    pats = [(1, s.encode()) for s, _ in rx]
    m = build(pats)
    exp = oracle.scan_patterns(pats, d)
    assert len(exp) >= 200 and np.array_equal(m.scan_array(d), exp)


@pytest.mark.parametrize("flags", [0, 3])
def test_tuned_matcher_keeps_its_prefixes(flags):
    # the tuner plans the groups anew: the covered ones are still not walked (no
    # chunk boundary is guessed)
    pats = [(1, rb"key=[0-9]+"), (1, rb"(?:alpha|beta1|gamma)[ :]{1,3}[a-f]{2,4}"), (1, rb"user_[a-z0-9_]*\.")]
    d = plant(text(1 << 20, 5), TEXTS, 97, 6)
    m = build(pats, max_matches=1 << 18, profile=True)
    exp = oracle.scan_patterns(pats, d)
    m.tune(text(1 << 20, 9), flags=flags)
    assert np.array_equal(m.scan_array(d), exp)
    assert m.info()["last_guesses"] == 0 and m.info()["last_events"] == 0
