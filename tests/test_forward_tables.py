"""The digit tables of the forward transforms as the kernels take them, decoded
on the host, and every transform table's level sums.

The stages are split radix-2 (decimation in frequency): a class holds the rows
(Re, Im) of its kept outputs over the first half of the inputs, which the
kernel gives as sums (even outputs) or differences (odd ones) of the two
halves; an odd padded z length keeps one class over all inputs.  The decoded
rows are compared with the DFT's definition, and with the folded halves of the
full transform of a random line.

A level sum of a chunk (two k-tiles; Grid::tcch for the inverse) has to stay
within +-(2^22 - 2^10) whatever the data's digits: |d| <= 128, the top one 256, or
512 for the sums and differences, which have 57 bits.
"""
import ctypes
import math
from pathlib import Path

import numpy as np
import pytest

from test_product_tc_tables import decode

LIB = Path(__file__).resolve().parent.parent / "shadow-channel_gb300" / "libc_channel.so"
GRIDS = [(16, 9, 16), (28, 9, 18), (12, 9, 14), (32, 9, 32), (48, 9, 48), (128, 9, 128), (24, 9, 98)]


@pytest.fixture(scope="module")
def lib():
    if not LIB.exists():
        import build
        build.build()
    L = ctypes.CDLL(str(LIB))
    L.c_setup_tc_table.argtypes = [ctypes.c_int] * 3 + [ctypes.c_double] * 5 + [
        ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p]
    return L


def table(lib, grid, which):
    args, sizes = (*grid, 2 * math.pi, math.pi, 2000.0, 2.0, 0.01, which), (ctypes.c_longlong * 2)()
    assert lib.c_setup_tc_table(*args, None, 0, None, 0, sizes) == 0
    frag, ex = np.zeros(sizes[0], np.uint32), np.zeros(sizes[1], np.int32)
    assert lib.c_setup_tc_table(*args, frag.ctypes.data, sizes[0], ex.ctypes.data, sizes[1], sizes) == 0
    return frag, ex


def classes(lib, grid, which, outs, K):
    """the decoded rows of each class"""
    frag, ex = table(lib, grid, which)
    KT, res, f0, e0 = (K + 15) // 16, [], 0, 0
    for out in outs:
        rows = 2 * len(out)
        MT = (rows + 15) // 16
        n = MT * KT * 7 * 32 * 4
        res.append(decode(frag[f0:f0 + n], ex[e0:e0 + rows], 1, MT, KT)[0][:, :K])
        f0, e0 = f0 + n, e0 + rows
    assert f0 == frag.size and e0 == ex.size
    return res


def z_modes(Nz, pz):
    zo = [k if k < Nz // 2 else k + 1 + Nz // 2 for k in range(Nz - 1)]
    if pz % 2:
        return [zo]
    return [[z for z in zo if z % 2 == c] for c in (0, 1)]


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_x_stage(lib, grid):
    Nx, _, Nz = grid
    px, pz, X = 3 * Nx // 2, 3 * Nz // 2, Nx // 2
    h, outs = px // 2, [list(range(c, X, 2)) for c in (0, 1)]
    rng = np.random.default_rng(0)
    p = rng.standard_normal(px)
    want = np.fft.fft(p)
    for which, norm in ((11, 1.0 / (px * pz)), (13, 1.0)):
        for c, (rows, kx) in enumerate(zip(classes(lib, grid, which, outs, h), outs)):
            ang = 2 * np.pi * (np.outer(kx, np.arange(h)) % px) / px
            ref = np.stack([np.cos(ang), -np.sin(ang)], 1).reshape(2 * len(kx), h) * norm
            assert np.abs(rows - ref).max() <= 4e-15 * norm  # as test_forward_dft_tables
            y = rows @ (p[:h] + p[h:] if c == 0 else p[:h] - p[h:])
            assert np.abs(y[0::2] + 1j * y[1::2] - norm * want[kx]).max() <= 1e-13 * norm * px


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_z_stage(lib, grid):
    _, _, Nz = grid
    pz = 3 * Nz // 2
    outs = z_modes(Nz, pz)
    h = pz // len(outs)
    rng = np.random.default_rng(1)
    y = rng.standard_normal(pz) + 1j * rng.standard_normal(pz)
    want = np.fft.fft(y)
    for c, (rows, zo) in enumerate(zip(classes(lib, grid, 12, outs, 2 * h), outs)):
        ang = 2 * np.pi * (np.outer(zo, np.arange(h)) % pz) / pz
        ref = np.zeros((2 * len(zo), 2 * h))
        ref[0::2, 0::2], ref[0::2, 1::2] = np.cos(ang), np.sin(ang)
        ref[1::2, 0::2], ref[1::2, 1::2] = -np.sin(ang), np.cos(ang)
        assert np.abs(rows - ref).max() <= 4e-15
        a = y if len(outs) == 1 else (y[:h] + y[h:] if c == 0 else y[:h] - y[h:])
        F = rows @ np.stack([a.real, a.imag], 1).ravel()
        assert np.abs(F[0::2] + 1j * F[1::2] - want[zo]).max() <= 1e-13 * pz


def digits(frag, MT, KT):
    """|digit| [7][rows][K] of a fragment table"""
    w = frag.reshape(MT, KT, 7, 32, 4)
    out = np.zeros((7, MT * 16, KT * 16), np.int64)
    lane = np.arange(32)
    g, t = lane >> 2, lane & 3
    for word, (dr, dk) in enumerate(((0, 0), (8, 0), (0, 8), (8, 8))):
        for half in (0, 1):
            bits = (w[..., word] & 0xFFFF0000) if half else (w[..., word] & 0xFFFF) << 16
            v = np.abs(np.ascontiguousarray(bits.astype(np.uint32)).view(np.float32)).astype(np.int64)
            for mt in range(MT):
                for kt in range(KT):
                    out[:, mt * 16 + g + dr, kt * 16 + 2 * t + dk + half] = v[mt, kt]
    return out


def worst_level(d, chunk, top):
    """the largest level sum that any data digits can reach over `chunk` k-tiles
    in a row"""
    K, worst = d.shape[2], 0
    for k0 in range(0, K, 16):
        s = d[:, :, k0:k0 + 16 * chunk].sum(2)  # of each digit over the window
        lower = np.concatenate([np.zeros((1, s.shape[1]), np.int64), np.cumsum(s, 0)[:-1]])
        worst = max(worst, int((128 * lower + top * s).max()))
    return worst


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_level_sums_stay_exact(lib, grid):
    Nx, _, Nz = grid
    px, pz, X = 3 * Nx // 2, 3 * Nz // 2, Nx // 2
    info = (ctypes.c_int * 4)()
    assert lib.c_setup_transform_rows(*grid, info) == 0
    assert info[0] in (2, 3) and info[1] >= 2  # the kernels' chunks: Grid::tcch, two
    limit = 2 ** 22 - 2 ** 10
    for which in (2, 3):  # the inverse's stages
        frag, ex = table(lib, grid, which)
        MT = (ex.size + 15) // 16
        d = digits(frag, MT, frag.size // (MT * 7 * 32 * 4))
        assert worst_level(d, info[0], 256) <= limit
    zs = z_modes(Nz, pz)
    xs = [list(range(c, X, 2)) for c in (0, 1)]
    for which, outs, K, top in ((11, xs, px // 2, 512), (13, xs, px // 2, 512),
                                (12, zs, 2 * pz // len(zs), 512 if len(zs) == 2 else 256)):
        frag, _ = table(lib, grid, which)
        KT, f0 = (K + 15) // 16, 0
        for out in outs:
            MT = (2 * len(out) + 15) // 16
            n = MT * KT * 7 * 32 * 4
            assert worst_level(digits(frag[f0:f0 + n], MT, KT), 2, top) <= limit
            f0 += n


def test_digits_of_sums_of_two_integers():
    """57-bit values: seven balanced digits, the top one within +-512"""
    S = sum(256 ** i for i in range(6))
    for x in (2 ** 57, -(2 ** 57), 2 ** 57 - 1, 512 * 256 ** 6 - 128 * S, 0, -1, 0x7F7F7F7F7F7F):
        word = (x + 0x6600808080808080) & (2 ** 64 - 1)  # the kernels' offset: 1536 + d_0 as fp16 bits, 128 + d_q
        top = ((word >> 48) & 0xFFFF) - 0x6600
        low = [((word >> (8 * k)) & 255) - 128 for k in range(5, -1, -1)]
        assert sum(v * 256 ** (6 - q) for q, v in enumerate([top] + low)) == x
        assert -512 <= top <= 512
        # fp16 0x6600 is 1536, one unit of the last place 1 from 1024 to 2048
        assert np.array([0x6600 + top], np.uint16).view(np.float16)[0] == 1536 + top
