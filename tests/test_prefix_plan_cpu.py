"""Which regexes the literal filter covers (host side): the choice of the prefix
length over pattern sets, by the planner's own code."""
import ctypes
import random

import pytest


def prefix_plan(literals, regexes, states=0, fold=False):
    """(prefix length, 0 for none; per regex whether it is covered)"""
    import warpstate_b200 as ws
    from warpstate_b200 import _native as N
    b = ws.PatternSet.builder().case_insensitive(fold)
    for x in literals:
        b = b.literal_bytes(x)
    for x in regexes:
        b = b.regex(x)
    ps = b.build()
    fn = N.lib().ws_testing_prefix_plan
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_uint, ctypes.c_char_p, ctypes.c_ulong]
    buf = ctypes.create_string_buffer(len(regexes) + 1)
    n = fn(ps._h, states, buf, len(regexes))
    assert n >= 0
    return n, [buf.raw[i] != 0 for i in range(len(regexes))]


def nucleotide_set(kmers, motifs, seed=3):
    r = random.Random(seed)
    lits = list({bytes(r.choices(b"ACGT", k=r.randint(20, 32))) for _ in range(kmers)})
    out = []
    for _ in range(motifs):  # one degenerate base each, 20 to 40 bases
        m = r.choices("ACGT", k=r.randint(20, 40))
        m[r.randrange(len(m))] = r.choice(["[AG]", "[CT]", "[ACGT]"])
        out.append("".join(m))
    return lits, out


SHORT = ["GT[CT][AG]AC", "G[CT]GGCC[AG]C", "GT[CT][AG]ACGGTAC[AT]", "GT[CT][AG]ACGGTAC[AT]ACGT", "AC[AG]TTGCAACGGTTACGT"]


@pytest.mark.parametrize("short", SHORT)
@pytest.mark.parametrize("motifs", [0, 40])
def test_short_motif_does_not_choose_the_layout(short, motifs):
    # beside k-mers, a motif of fewer than 19 bases is walked: 16-byte grams stay
    # possible for the others
    lits, rx = nucleotide_set(5000, motifs)
    n, covered = prefix_plan(lits, rx + [short])
    assert covered == [True] * motifs + [False]
    assert n == (20 if motifs else 0)


@pytest.mark.parametrize("size", [19, 20])
def test_motif_of_nineteen_bases_is_covered(size):
    lits, rx = nucleotide_set(5000, 3)
    assert prefix_plan(lits, rx + [("AC[AG]" + "TTGCAACGGTTACGTACG")[:size + 3]]) == (20, [True] * 4)


def test_motif_with_too_many_prefixes_is_walked_alone():
    lits, rx = nucleotide_set(5000, 10)
    wide = "ACGT" + "[ACGT]" * 6 + "TTGCAACGGTTACGT"  # 4,096 strings of 20 bases, above the limit of one regex
    assert prefix_plan(lits, rx + [wide]) == (20, [True] * 10 + [False])


def test_short_kmer_keeps_every_motif_walked():
    lits, rx = nucleotide_set(5000, 10)
    assert prefix_plan(lits + [b"ACGTACGTACGT"], rx) == (0, [False] * 10)


def test_sets_over_letters_are_covered_at_their_length():
    words = [r"alpha[0-9]{1,3}x", r"(?:gamma|delta)=[a-f]+", r"tailwind [0-9]"]
    assert prefix_plan([], words) == (7, [True] * 3)
    assert prefix_plan([], words + [r"[0-9]+px"])[1] == [True] * 3 + [False]
    assert prefix_plan([], [r"[0-9]+px"]) == (0, [False])


def sharing(n, head, seed=8):
    r = random.Random(seed)
    tails = set()
    while len(tails) < n:
        tails.add("".join(r.choices("abcdefghij", k=r.randint(5, 10))))
    return [f"{head}{t}/[a-z0-9]{{1,6}}" for t in sorted(tails)]


@pytest.mark.parametrize("n", [1, 24, 25, 300])
def test_regexes_that_share_a_beginning(n):
    # up to 24 regexes are walked in turn from a beginning they share; more of
    # them are left to their groups' walk, the others stay with the filter
    rx = [r"alpha[0-9]{1,3}x", r"tailwind [0-9]", r"key=[0-9]+"]
    got, covered = prefix_plan([], sharing(n, "http://www.") + rx)
    assert got > 0 and covered == [n <= 24] * n + [True] * 3
    # a shorter beginning of the same words counts with the longer ones
    got, covered = prefix_plan([], sharing(n, "http://www.") + rx + ["http[0-9s]*:", "http:[/]?x"])
    assert covered[:n] == [n + 1 <= 24] * n and covered[n:n + 3] == [True] * 3


def test_regexes_with_beginnings_of_their_own_are_all_covered():
    assert prefix_plan([], joined_words(400))[1] == [True] * 400


def joined_words(n):
    r = random.Random(12)
    return ["".join(r.choices("abcdefghijklmnop", k=9)) + "[0-9]{1,4}x" for _ in range(n)]


@pytest.mark.parametrize("n", [20, 70])
def test_buckets_by_four_bytes_stay_short(n):
    # n beginnings of 8 bytes with the same first 4, and one regex whose own has
    # only 4: it would make the table's buckets go by 4 bytes
    rx = ["user" + "".join(chr(97 + (i // 5 ** k) % 5) for k in range(4)) + "[0-9]{1,3};" for i in range(n)]
    got, covered = prefix_plan([], rx + [r"abcd[0-9a-f]+;"])
    assert covered[:n] == [True] * n and covered[n] == (n <= 64)


def test_literals_with_long_grams_decide():
    # '=' and digits at the ends of the prefixes do not make nucleotide literals
    # sparse: those of 11 bytes and more keep their long grams
    r = random.Random(4)
    lits = sorted({bytes(r.choices(b"ACGT", k=r.randint(12, 16))) for _ in range(4000)})
    rx = ["".join(r.choices("ACGT", k=r.randint(4, 7))) + "=[0-9]+" for _ in range(15)]
    assert prefix_plan(lits, rx) == (0, [False] * 15)
    assert prefix_plan(lits[::100], rx) == (0, [False] * 15)
    assert prefix_plan([b"needle", b"haystack"], rx)[1] == [True] * 15
    assert prefix_plan([], rx)[1] == [True] * 15


@pytest.mark.parametrize("letters", ["abcdefgh", "abcdefghijkl"])
def test_short_words_over_few_letters_are_covered(letters):
    # (by the compacting kernel: their grams crowd the alphabet, their beginnings
    # do not fill the list)
    r = random.Random(6)
    rx = sorted({"\\b" + "".join(r.choices(letters, k=r.randint(5, 9))) + "\\b" for _ in range(60)})
    assert all(prefix_plan([], rx)[1])


def test_one_byte_literals_leave_the_list_to_themselves():
    rx = [r"alpha[0-9]{1,3}x", r"tailwind [0-9]"]
    assert prefix_plan([b"q", b"needle"], rx) == (0, [False] * 2)
    assert prefix_plan([b"qz", b"needle"], rx)[1] == [True] * 2
