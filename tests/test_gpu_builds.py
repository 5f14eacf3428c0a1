"""The kernels' builds for few blocks, large planes and odd sizes against the
FP64 kernels (CHN_RECON_FP64=1, CHN_TRANSFORMS_FP64=1; past their shared
memory, Ny > 160, the digit GEMMs in the builds of many blocks:
CHN_SOLVE_TILE=16, CHN_RECON_BUILD=0).

One step each way of a small batch: primal, tangents (one forced), coupled and
exact adjoint.  The grids sit where a build begins or ends:

- few-block reconstruction, solve and transposed solve: Ny - 2 = 16, 17
  coefficient rows (the reconstruction's lower end), 65 (a second row pair per
  thread), 129 (past its upper end), 171 (past the solve's shared
  memory), 6 kx columns (a partial tile of 4), and more tiles than the build
  takes;
- forward transforms split radix-2: an odd padded z length (one class), class
  lengths with remainders, 60x33x48 (two k-tiles per digit sum);
- components in blocks of their own (one trajectory at 32x65x32) and together
  (20x17x18, 20 trajectories: three product planes per pass);
- 48x33x48, 10 trajectories: the inverse's x stage in chunks, one product plane
  a pass in the wider blocks;
- planes that do not fit one block: 128x33x64, and 128x33x54 (odd).

Both evaluate the same step to rounding.  The oracle built with and without
FMA contraction differs by at most (primal, tangent, adjoint) 1.2e-12, 2.4e-12,
3.0e-12 on these grids with Ny <= 33, 8.8e-12, 1.5e-11, 2.8e-11 to Ny = 67,
4.3e-10, 9.4e-10, 7.8e-10 to 131 and 3.9e-9, 3.9e-9, 3.1e-9 to 172: twice that
(at least the one-step parity tolerances 5e-12, 1e-11, 3e-11).
"""
import ctypes
import os

import numpy as np
import pytest

import oracle as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu

TOL = [(33, (5e-12, 1e-11, 3e-11)), (67, (1.8e-11, 3e-11, 5.6e-11)), (131, (8.6e-10, 1.9e-9, 1.6e-9)),
       (172, (7.8e-9, 7.8e-9, 6.2e-9))]
CASES = [(12, 18, 6, 1, 2), (12, 19, 6, 1, 2), (20, 67, 6, 2, 2), (12, 131, 6, 1, 2), (12, 171, 6, 1, 1),
         (20, 33, 16, 12, 2), (20, 17, 18, 20, 2), (32, 65, 32, 1, 1), (60, 33, 48, 1, 1),
         (48, 33, 48, 10, 1), (128, 33, 64, 1, 1), (128, 33, 54, 2, 1)]


def _step(cc, Nx, Ny, Nz, nseg, ntan, ref):
    names = ("CHN_RECON_FP64", "CHN_TRANSFORMS_FP64", "CHN_SOLVE_TILE", "CHN_RECON_BUILD", "CHN_AUTOTUNE")
    old = {k: os.environ.pop(k, None) for k in names}
    os.environ["CHN_AUTOTUNE"] = "0"
    if ref and Ny <= 160:
        os.environ.update({"CHN_RECON_FP64": "1", "CHN_TRANSFORMS_FP64": "1"})
    elif ref:
        os.environ.update({"CHN_SOLVE_TILE": "16", "CHN_RECON_BUILD": "0"})
    try:
        assert cc.c_init(Nx, Ny, Nz, 2 * np.pi, np.pi, 2000.0, 2.0, 0.004, 1) == 0, cc.c_last_error_message()
        lib = cc.lib
        assert lib.c_batch_init(nseg, ntan, ntan - 1) == 0, cc.c_last_error_message()
        try:
            C = np.stack([O.synthetic_state(Nx, Ny, Nz, seed=s) for s in range(nseg)])
            IC = np.stack([np.stack([O.synthetic_state(Nx, Ny, Nz, seed=100 + ntan * s + j, laminar=False)
                                     for j in range(ntan)]) for s in range(nseg)])
            AC = np.stack([O.synthetic_state(Nx, Ny, Nz, seed=200 + s, laminar=False) for s in range(nseg)])
            AX = AC.copy()
            inh = (ctypes.c_int * ntan)(*([0] * (ntan - 1) + [1]))
            assert lib.c_batch_forward(0, 1, C.ctypes.data, IC.ctypes.data, inh) == 0, cc.c_last_error_message()
            assert lib.c_batch_adjoint(1, 0, AC.ctypes.data, 1.0) == 0, cc.c_last_error_message()
            if Ny <= 131:   # its blocks' shared memory ends near Ny = 160
                assert lib.c_batch_adjoint_exact(1, 0, AX.ctypes.data) == 0, cc.c_last_error_message()
        finally:
            lib.c_batch_destroy()
        cc.c_destroy()
        return (C, IC, AC, AX) if Ny <= 131 else (C, IC, AC)
    finally:
        for k, v in old.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
def test_builds_match_the_fp64_kernels(case):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    tc, ref = _step(cc, *case, False), _step(cc, *case, True)
    tp, tt, ta = next(t for ny, t in TOL if case[1] <= ny)
    for a, b, tol in zip(tc, ref, (tp, tt, ta, ta)):
        if case[1] <= 160:
            assert not np.array_equal(a, b)   # two builds' roundings, not one's
        for s in range(a.shape[0]):
            assert np.linalg.norm(a[s] - b[s]) <= tol * np.linalg.norm(b[s])


def test_uneven_batch_of_odd_and_even_padded_lengths():
    """3 Nz/2 = 21 beside 18, whose z-stage digits need a k-tile more: each
    instance against itself alone."""
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    grids = [(12, 17, 14), (12, 17, 12), (12, 17, 14)]
    i3 = lambda j: (ctypes.c_int * 3)(*[g[j] for g in grids])
    d3 = lambda v: (ctypes.c_double * 3)(v, v, v)
    states = [[O.synthetic_state(*g, seed=k + i, laminar=k == 0) for i, g in enumerate(grids)] for k in (0, 10, 20)]
    C, IC, AC = (np.concatenate([x.ravel() for x in xs]) for xs in states)
    inh = (ctypes.c_int * 1)(1)
    assert cc.lib.c_multi_init(3, i3(0), i3(1), i3(2), d3(2 * np.pi), d3(np.pi), d3(2000.0), d3(2.0), d3(0.004), 1, 1,
                               0) == 0, cc.c_last_error_message()
    try:
        assert cc.lib.c_multi_forward(0, 1, C.ctypes.data, IC.ctypes.data, inh) == 0, cc.c_last_error_message()
        assert cc.lib.c_multi_adjoint(1, 0, AC.ctypes.data, 1.0) == 0, cc.c_last_error_message()
    finally:
        cc.lib.c_multi_destroy()
    off = 0
    for i, g in enumerate(grids):
        c, ic, ac = (states[k][i].copy() for k in range(3))
        assert cc.c_init(*g, 2 * np.pi, np.pi, 2000.0, 2.0, 0.004, 1) == 0, cc.c_last_error_message()
        cc.c_primal(0, c)
        cc.c_tangent(0, 1, ic, 1)
        cc.c_adjoint(1, 0, ac, 0, 1.0)
        assert cc.c_last_error() == 0, cc.c_last_error_message()
        cc.c_destroy()
        for a, b, tol in zip((C, IC, AC), (c, ic, ac), TOL[0][1]):
            assert np.linalg.norm(a[off:off + b.size] - b.ravel()) <= tol * np.linalg.norm(b)
        off += c.size
