"""The limits of a regex's prefix lists, and that counting the paths before they
are spelled out keeps them (host side)."""
import itertools
import time

import pytest

from test_prefix_cpu import prefixes


@pytest.mark.parametrize("most", [999, 1000, 1001])
def test_limit_is_exact(most):
    got = prefixes(r"abcd[0-9]{3}z", 7, most)
    # (one byte continues: the strings go on to 8 bytes)
    want = sorted(("abcd" + "".join(t) + "z").encode() for t in itertools.product("0123456789", repeat=3))
    assert got == (want if most >= 1000 else -1)


def test_strings_of_different_ends():
    assert prefixes(r"abcd(?:e|fg|hij[kl]m)?", 20) == [b"abcd"]
    assert prefixes(r"(?:abcde|abcdfg|abchij[kl]m)x", 20) == [b"abcdex", b"abcdfgx", b"abchijkmx", b"abchijlmx"]


def test_starts_of_every_left_context_count_once():
    assert prefixes(r"(?:^|\b)abcd[01]", 5) == [b"abcd0", b"abcd1"]
    assert len(prefixes(r"\bkey[0-9]{2}x", 6, 100)) == 100


def test_too_many_strings_are_counted_not_spelled():
    t = time.time()
    for _ in range(20):
        assert prefixes(r"(?:abcd|bcde|cdef)[a-p]{1,8}(?:xyz[a-p]{4}|zyx[a-p]{4})[0-9]{1,9}", 20, 2048) == -1
    assert time.time() - t < 2
