"""Required prefixes of a regex (host side): every match begins with exactly one
listed prefix, whatever the left and right context, and the limits hold."""
import ctypes
import random

import pytest

import oracle

# source, prefix length, a text that holds a match
CASES = [
    (r"(?:abcd|abxyz|q1234)[0-9]{1,8}(?:zz|y)", 5, b"abcd77y"),
    (r"key=[0-9]+", 7, b"key=1"),
    (r"(?:http|https)://[a-z]+\.[a-z]{2}", 7, b"https://a.bc"),
    (r"abcd|abcde|abcdef", 7, b"abcdef"),
    (r"\b(?:fatal|error|warn!)\b", 7, b" fatal."),
    (r"^GET [^ ]{1,4} HTTP", 4, b"\nGET /a HTTP"),
    (r"end of (?:file|line)$", 5, b"end of line\n"),
    (r"(?i)error: [a-f]", 7, b"ErRor: a"),
    (r"a[bc]{2}d+e?", 4, b"abcdde"),
    (r"[ACGT]{2}ACGTTGCA[AG]CCGTTGCAAC", 20, b"TTACGTTGCAACCGTTGCAAC"),
    (r"x\x00y\xffz.", 5, b"x\x00y\xffzq"),
]


def prefixes(source, length, most=4096):
    from warpstate_b200 import _native as N
    fn = N.lib().ws_testing_regex_prefixes
    fn.restype = ctypes.c_long
    fn.argtypes = [ctypes.c_char_p, ctypes.c_uint, ctypes.c_ulong, ctypes.c_char_p, ctypes.c_ulong]
    buf = ctypes.create_string_buffer(1 << 20)
    n = fn(source.encode(), length, most, buf, len(buf))
    if n < 0:
        return n
    out = [bytes.fromhex(x) for x in buf.value.decode().split()]
    assert len(out) == n
    return out


@pytest.mark.parametrize("source,length,sample", CASES)
def test_every_match_begins_with_one_prefix(source, length, sample):
    found = prefixes(source, length)
    assert isinstance(found, list) and found
    assert all(len(p) >= 4 for p in found)
    for a in found:
        assert not any(b != a and a.startswith(b) for b in found)
    # random text made of the regex's own prefixes and pieces, matched by the oracle
    r = random.Random(len(source))
    letters = sorted(set(b"".join(found)) | set(b" \nabz0=."))
    seen = 0
    for _ in range(3000):
        t = bytes(r.choices(letters, k=r.randint(0, 3))) + r.choice([sample] + found[:200]) + \
            bytes(r.choices(letters, k=r.randint(0, 12)))
        for s, e in oracle.Regex(source).find_iter(t):
            assert sum(t.startswith(p, s) for p in found) == 1, (t, s, e)
            seen += 1
    assert list(oracle.Regex(source).find_iter(sample)) and seen > 0


@pytest.mark.parametrize("source,why", [
    (r"abc|abcd", "a match of 3 bytes"), (r"[a-z]{1,8}q", "too many"), (r"\w+@x", "too many"), (r"ab$", "short"),
    (r".*abcd", "any first byte"), (r"(?:ab)+", "a match of 2 bytes"),
])
def test_regexes_without_prefixes(source, why):
    assert prefixes(source, 4, 512) == -1, why


def test_limit_counts_prefixes():
    assert len(prefixes(r"abcd[0-9][0-9]", 6, 100)) == 100
    assert prefixes(r"abcd[0-9][0-9]", 6, 99) == -1
    assert len(prefixes(r"abcd[0-9][0-9]", 4, 1)) == 1
