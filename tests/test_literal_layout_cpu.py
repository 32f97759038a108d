"""The literal filter's layout for a set (host side): the gram kernel only for sets
whose survivors on an input over their own letters fit its list."""
import ctypes
import random

import pytest

LOWER = b"abcdefghijklmnopqrstuvwxyz"


def layout(literals):
    import warpstate_b200 as ws
    from warpstate_b200 import _native as N
    b = ws.PatternSet.builder()
    for x in literals:
        b = b.literal_bytes(x)
    ps = b.build()
    fn = N.lib().ws_testing_literal_layout
    fn.restype, fn.argtypes = None, [ctypes.c_void_p, ctypes.c_void_p]
    out = (ctypes.c_uint * 3)()
    fn(ps._h, out)
    return out[0], out[1], bool(out[2])


def words(letters, n, shortest, longest=14, seed=3):
    r = random.Random(seed)
    return sorted({bytes(r.choices(LOWER[:letters], k=r.randint(shortest, longest))) for _ in range(n)})


@pytest.mark.parametrize("letters,n,shortest,period,gram,kernel", [
    (8, 45, 8, 4, 4, True), (8, 60, 8, 4, 4, False), (8, 200, 8, 4, 4, False), (12, 230, 8, 4, 4, True),
    (12, 320, 8, 4, 4, False), (26, 5000, 8, 4, 4, True), (26, 10_000, 8, 4, 4, False), (26, 28_000, 8, 4, 4, False),
    (26, 3500, 5, 2, 4, True), (26, 5000, 5, 2, 4, False), (26, 5500, 4, 1, 4, True), (26, 6000, 4, 1, 4, False),
    (26, 180, 3, 1, 3, True), (26, 250, 3, 1, 4, False),
])
def test_gram_kernel_for_sparse_sets(letters, n, shortest, period, gram, kernel):
    assert layout(words(letters, n, shortest)) == (period, gram, kernel)


def test_long_grams_for_small_alphabets():
    assert layout(words(4, 5000, 20, 32)) == (4, 16, True)
    assert layout(words(4, 5000, 12, 18)) == (4, 8, False)
    assert layout(words(4, 5000, 12, 18) + [b"ab"]) == (4, 8, False)
