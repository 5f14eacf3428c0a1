"""The sums of the digit GEMMs (csrc/digit_sum.cuh), the library's own code
run on the host against Python integers.

A contraction's level sums, chunk by chunk, fold into t 2^s + r, which has to
be the exact sum in units of level 6 for any level sums within the
accumulators' range of +-2^22 (less what r adds): no chunk rounds anything
off.  The word that is converted to FP64 has to give that sum correctly
rounded, for one contraction and for the sum and difference of two (s = 8), or
cut to four units first (s = 10, which has room for long rows).

A sum that is kept between a transform's stages gives its column an exponent
field: that of a NaN past FP64's range (a larger number would pass for a finite
one, and hide a NaN beside it).

A table's row exponents have to be those of its entries, whatever the row's
length: a larger one gives away table bits.
"""
import ctypes
import math
import random
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

LIB = Path(__file__).resolve().parent.parent / "shadow-channel_gb300" / "libc_channel.so"
TOP = 2 ** 22 - 2 ** 10


@pytest.fixture(scope="module")
def lib():
    if not LIB.exists():
        import build
        build.build()
    L = ctypes.CDLL(str(LIB))
    L.c_setup_digit_sum.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                                    ctypes.c_int, ctypes.c_void_p]
    return L


def fold(lib, shift, a, b=(), op=0, first=0):
    ia, ib = ((ctypes.c_int * max(1, 7 * len(x)))(*[v for c in x for v in c]) for x in (a, b))
    out = (ctypes.c_longlong * 4)()
    assert lib.c_setup_digit_sum(shift, ia, len(a), ib, len(b), op, first, out) == 0  # both forms of the fold agree
    return tuple(out)


def exact(chunks):
    return sum(v * 256 ** (6 - l) for c in chunks for l, v in enumerate(c))


def chunks(rng, n, scale, shift, parts=1):
    """level sums: extremes, small ones (cancelling high levels), any; level 0,
    whose total the tables' row exponents bound, shared by the chunks (s = 8)"""
    kind = rng.randrange(4)
    top = [TOP // (n * parts) if shift == 8 else TOP] + [TOP] * 6
    if kind == 0:
        return [[rng.choice((-t, t)) // scale for t in top] for _ in range(n)]
    lead = rng.randrange(7) if kind == 1 else 0
    return [[0 if l < lead else rng.randint(-t, t) // scale for l, t in enumerate(top)] for _ in range(n)]


@pytest.mark.parametrize("shift,n", [(8, 1), (8, 2), (8, 3), (8, 5), (8, 16), (10, 1), (10, 2), (10, 4)])
def test_a_fold_keeps_the_whole_sum(lib, shift, n):
    rng = random.Random(n)
    for _ in range(2000):
        a = chunks(rng, n, rng.choice((1, 16, 1024)), shift)
        first = rng.choice((0, 128))
        t, r, _, _ = fold(lib, shift, a, first=first)
        assert 0 <= r < 2 ** shift
        assert t * 2 ** shift + r == exact(a) + first


@pytest.mark.parametrize("shift,op", [(8, 0), (8, 1), (8, 2), (10, 0), (10, 1), (10, 2)])
def test_the_rounded_word(lib, shift, op):
    """x 2^(s - up) to FP64: within half a unit in the last place of the sum
    (s = 10: of the sum less its remainder by 4)"""
    rng = random.Random(100 + op)
    for _ in range(4000):
        n = rng.randint(1, 6 if shift == 8 else 2)
        a, b = (chunks(rng, n, rng.choice((1, 64)), shift, 2) for _ in range(2))
        if rng.random() < 0.3:  # nearly equal parts: differences of every size
            b = [[v + (rng.randint(-3, 3) if l >= rng.randrange(8) else 0) for l, v in enumerate(c)] for c in a]
            top = [TOP // (2 * n) if shift == 8 else TOP] + [TOP] * 6
            b = [[max(-t, min(t, v)) for v, t in zip(c, top)] for c in b]
        want = exact(a) + (0, exact(b), -exact(b))[op]
        t, r, word, up = fold(lib, shift, a, b, op)
        assert t * 2 ** shift + r == want and r < 2 ** (shift + 1)
        assert -2 ** 63 <= word < 2 ** 63
        got = Fraction(float(word)) * Fraction(2) ** (shift - up)
        if shift == 10 and abs(t) < 2 ** 54:
            want -= want % 4
        lo = max(abs(want).bit_length() - 53, 0)
        assert abs(got - want) * 2 <= 2 ** lo
        if lo == 0:
            assert got == want


def tables(lib, grid, which):
    lib.c_setup_tc_table.argtypes = [ctypes.c_int] * 3 + [ctypes.c_double] * 5 + [
        ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p]
    args, sizes = (*grid, 2 * math.pi, math.pi, 2000.0, 2.0, 0.01, which), (ctypes.c_longlong * 2)()
    assert lib.c_setup_tc_table(*args, None, 0, None, 0, sizes) == 0
    ex = np.zeros(sizes[1], np.int32)
    assert lib.c_setup_tc_table(*args, None, 0, ex.ctypes.data, sizes[1], sizes) == 0
    return ex


@pytest.mark.parametrize("ny", [33, 129, 133, 179])
def test_legendre_row_exponents(lib, ny):
    """tables 0, 7: the bases [Q] and their transposes [R]; Rp's rows sum past
    127 of their scale from Ny = 133 on"""
    args = (4, ny, 4, 2 * math.pi, math.pi, 2000.0, 2.0, 0.01)
    lib.c_setup_table.argtypes = [ctypes.c_int] * 3 + [ctypes.c_double] * 5 + [ctypes.c_int, ctypes.c_void_p,
                                                                               ctypes.c_int]
    q, r, d = 3 * ny // 2, ny - 2, ny - 4
    ex, ext = tables(lib, (4, ny, 4), 0).reshape(5, q), tables(lib, (4, ny, 4), 7).reshape(5, r)
    for b, cols in enumerate((d, d, d, r, r)):
        m = np.zeros(q * cols)
        assert lib.c_setup_table(*args, b, m.ctypes.data, m.size) == m.size
        m = np.abs(m.reshape(q, cols))
        for e, rows in ((ex[b], m.max(1)), (ext[b][:cols], m.max(0))):
            live = rows > 0
            assert np.array_equal(e[live], np.frexp(rows[live])[1])


@pytest.mark.parametrize("nz", [128, 196, 256])
def test_long_transforms_have_tables(lib, nz):
    """the inverse z stage: rows of 2 (Nz - 1) entries of at most 1"""
    assert (tables(lib, (8, 17, nz), 2) == 1).all()


@pytest.mark.parametrize("t,e,ce,field", [
    (0, 900, 1023, 0), (1, 0, 1023, 1023), (-1, 0, 1023, 1023), (2 ** 40, 0, 1023, 1063), (3, -1100, 5, 1),
    (1, 1023, 2046, 2046), (1, 1024, 2046, 0x7FF), (2 ** 60, 972, 2046, 0x7FF), (-2 ** 60, 1030, 2046, 0x7FF),
    (7, 0, 0x7FF, 0x7FF), (0, 0, 0x7FF, 0x7FF)])
def test_exponent_field_of_a_kept_sum(lib, t, e, ce, field):
    lib.c_setup_sum_field.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    assert lib.c_setup_sum_field(t, e, ce) == field


@pytest.mark.parametrize("nx,nz,inverse,forward", [
    (16, 16, 0, 0), (32, 32, 0, 0), (48, 48, 0, 0), (24, 98, 0, 0), (12, 126, 0, 0), (8, 128, 0, 0), (84, 8, 0, 0), (128, 8, 0, 1),
    (8, 144, 0, 1), (144, 8, 0, 1), (8, 200, 1, 1)])
def test_which_transforms_have_long_rows(lib, nx, nz, inverse, forward):
    """(odd padded lengths, whose forward inputs are no sums of two, take twice
    the length)"""
    out = (ctypes.c_int * 4)()
    assert lib.c_setup_transform_rows(nx, 9, nz, out) == 0
    assert out[0] >= 2 and out[1] >= 2
    assert (out[2], out[3]) == (inverse, forward)
