"""The forward x table's kx = 0 row has equal entries, 1 / (px pz), whose digits
may all be large.  A long row (Nx from 88 on) whose digits would not allow two
k-tiles per chunk gives up a bit instead of turning the tensor-core
transforms off."""
import ctypes
from pathlib import Path

import pytest

LIB = Path(__file__).resolve().parent.parent / "shadow-channel_gb300" / "libc_channel.so"


@pytest.mark.parametrize("nx", [88, 96, 100, 108, 112, 120, 128, 144])
def test_long_rows_allow_two_k_tiles(nx):
    if not LIB.exists():
        import build
        build.build()
    lib = ctypes.CDLL(str(LIB))
    out = (ctypes.c_int * 4)()
    for nz in (8, 10, 12, 14, 16, 18, 20, 24, 28, 30, 32, 36, 40):
        assert lib.c_setup_transform_rows(nx, 9, nz, out) == 0
        assert out[1] >= 2, (nx, nz)
