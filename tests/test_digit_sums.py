"""The sums of the digit GEMMs (csrc/digit_sum.cuh), the library's own code
run on the host against Python integers.

A contraction's level sums, chunk by chunk, fold into t 2^s + r, which has to
be the exact sum in units of level 6 for any level sums within the
accumulators' range of +-2^22 (less what r adds): no chunk rounds anything
off.  The word that is converted to FP64 has to give that sum correctly
rounded, for one contraction and for the sum and difference of two.
"""
import ctypes
import random
from fractions import Fraction
from pathlib import Path

import pytest

LIB = Path(__file__).resolve().parent.parent / "shadow-channel_gb300" / "libc_channel.so"
TOP = 2 ** 22 - 2 ** 10


@pytest.fixture(scope="module")
def lib():
    if not LIB.exists():
        import build
        build.build()
    L = ctypes.CDLL(str(LIB))
    L.c_setup_digit_sum.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                                    ctypes.c_int, ctypes.c_void_p]
    return L


def fold(lib, a, b=(), op=0, first=0):
    ia, ib = ((ctypes.c_int * max(1, 7 * len(x)))(*[v for c in x for v in c]) for x in (a, b))
    out = (ctypes.c_longlong * 4)()
    shift = lib.c_setup_digit_sum(ia, len(a), ib, len(b), op, first, out)
    assert shift > 0  # the fold of bit patterns and that of integers agree
    return shift, *out


def exact(chunks):
    return sum(v * 256 ** (6 - l) for c in chunks for l, v in enumerate(c))


def chunks(rng, n, scale, parts=1):
    """level sums: extremes, small ones (cancelling high levels), any; level 0,
    whose total the tables' row exponents bound, shared by the chunks"""
    kind = rng.randrange(4)
    top = [TOP // (n * parts)] + [TOP] * 6
    if kind == 0:
        return [[rng.choice((-t, t)) // scale for t in top] for _ in range(n)]
    lead = rng.randrange(7) if kind == 1 else 0
    return [[0 if l < lead else rng.randint(-t, t) // scale for l, t in enumerate(top)] for _ in range(n)]


@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 16])
def test_a_fold_keeps_the_whole_sum(lib, n):
    rng = random.Random(n)
    for _ in range(2000):
        a = chunks(rng, n, rng.choice((1, 16, 1024)))
        first = rng.choice((0, 128))
        shift, t, r, _, _ = fold(lib, a, first=first)
        assert 0 <= r < 2 ** shift
        assert t * 2 ** shift + r == exact(a) + first


@pytest.mark.parametrize("op", [0, 1, 2])
def test_the_rounded_word(lib, op):
    """x 2^(s - up) to FP64: within half a unit in the last place of the sum"""
    rng = random.Random(100 + op)
    for _ in range(4000):
        n = rng.randint(1, 6)
        a, b = (chunks(rng, n, rng.choice((1, 64)), 2) for _ in range(2))
        if rng.random() < 0.3:  # nearly equal parts: differences of every size
            b = [[v + (rng.randint(-3, 3) if l >= rng.randrange(8) else 0) for l, v in enumerate(c)] for c in a]
            b = [[max(-t, min(t, v)) for v, t in zip(c, [TOP // (2 * n)] + [TOP] * 6)] for c in b]
        want = exact(a) + (0, exact(b), -exact(b))[op]
        shift, t, r, word, up = fold(lib, a, b, op)
        assert t * 2 ** shift + r == want and r < 2 ** (shift + 1)
        assert -2 ** 63 <= word < 2 ** 63
        got = Fraction(float(word)) * Fraction(2) ** (shift - up)
        lo = max(abs(want).bit_length() - 53, 0)
        assert abs(got - want) * 2 <= 2 ** lo
        if lo == 0:
            assert got == want
