"""Regexes that share the beginning their matches are found by, against the
oracle: as many as the filter covers, one more, and inputs on which walking them
all is more work than the filter takes on."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

HEAD = "http://www.shared-by-all.org/"


def rules(n):
    return [f"{HEAD}{chr(97 + i % 26)}{chr(97 + i // 26)}[0-9]{{1,3}}".encode() for i in range(n)] + [rb"key=[0-9]+"]


def scan(pats, data, **cfg):
    import warpstate_b200 as ws
    b = ws.PatternSet.builder()
    for p in pats:
        b = b.regex(p.decode())
    m = ws.GpuMatcher.with_config(b.build(), ws.AutoMatcherConfig().max_matches(1 << 20).profile(True))
    return m.scan_array(data), m.info()


@pytest.mark.parametrize("n", [24, 25, 200])
@pytest.mark.parametrize("size", [300, 5000, 1 << 20])
def test_shared_beginnings(n, size):
    r = np.random.default_rng(size)
    tails = ["aa1 ", "ba77;", "ca", "xa9999", "zz1", "/", "ac12x"]
    text = b"".join((HEAD + tails[int(r.integers(0, 7))]).encode() + b"-" * int(r.integers(0, 400)) + b"key=9 "
                    for _ in range(max(2, size // 240)))[:size]
    pats = rules(n)
    d = np.frombuffer(text, dtype=np.uint8)
    got, info = scan(pats, d)
    exp = oracle.scan_patterns([(1, p) for p in pats], d)
    assert len(exp) >= 1 and np.array_equal(got, exp)
    assert info["n_groups"] >= (1 if n <= 24 else 2)


@pytest.mark.parametrize("every,gives_up", [(72, True), (1500, False)])
def test_work_of_many_short_walks_is_bounded(every, gives_up):
    # 24 walks of 30 bytes at one position in 72 bytes: the groups' walk takes over
    # (it finds match events; the filter's candidates need none)
    pats = rules(24)
    unit = [(HEAD + t).encode() for t in ("aa1", "b", "xa22", "//")]
    text = b"".join(u + b"." * (every - len(u)) for u in unit)
    d = np.frombuffer(text * ((24 << 20) // len(text)), dtype=np.uint8)
    got, info = scan(pats, d)
    exp = oracle.scan_patterns([(1, p) for p in pats], d)
    assert len(exp) == 2 * (len(d) // len(text)) and np.array_equal(got, exp)
    assert (info["last_events"] > 0) == gives_up
