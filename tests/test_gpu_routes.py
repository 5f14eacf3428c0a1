"""Calls whose kernels a rule picks, against the kernels of another rule.

Long transforms: 144x17x8 and 8x17x144, whose forward tables' rows have no room in
the sums that other grids keep between the stages, run the one-block products
with coarser ones, 8x17x200 the FFT kernels.  They agree with the FP64 kernels to
rounding (the oracle built with and without FMA contraction differs by at most
3.3e-13, 4.0e-13, 3.4e-13 in primal, tangent and adjoint there; the one-step parity
tolerances hold), and the products' builds with one another bit for bit.

A flow without spanwise variation whose spanwise velocity is 1e-10 of the
streamwise one: w and the wall-normal vorticity, odd under spanwise reflection,
keep their own relative accuracy through a step, in every build (the (0, 0)
line's u and w are two columns of one contraction, with an exponent each).  The
odd part alone (beta of kz = 0) is compared; the oracle built with and without
FMA contraction differs in it by 7.5e-13, 6.3e-13, 8.8e-13 and (exact adjoint)
1.3e-13, and the parity tolerances hold for it too.

The adjoint's two product passes as concurrent branches, which only launches of
more than two planes an SM are (4 of 32x65x32, 7 of 16x33x16, 3 of 48x97x48),
and products of one component a block, which launches of fewer are, give the
bits of the passes in turn and of whole planes a block.

Uneven batches whose largest padded z length is odd: 147 beside 18 (24x17x98 and
20x17x12) keeps the tensor-core transforms, 21 beside 18 (12x17x14 and 20x17x12)
is sized for an instance that needs more shared memory than the largest, 216 x
12 beside 18 (144x17x8, long rows) takes the coarser sums for all.  Each
instance against itself alone; the oracle's two builds differ by at most
3.9e-13 there.
"""
import ctypes
import os

import numpy as np
import pytest

import oracle as O
from conftest import has_gpu
import test_gpu_variants as V
from test_gpu_builds import _step

pytestmark = pytest.mark.gpu

PARITY = (5e-12, 1e-11, 3e-11, 3e-11)  # primal, tangent, adjoint, exact adjoint


@pytest.mark.parametrize("case", [(144, 17, 8, 1, 2), (8, 17, 144, 1, 2), (8, 17, 144, 4, 2), (8, 17, 200, 1, 2)],
                         ids=lambda c: "x".join(map(str, c)))
def test_long_transforms_match_the_fp64_kernels(case):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    for a, b, tol in zip(_step(cc, *case, False), _step(cc, *case, True), PARITY):
        for s in range(a.shape[0]):
            assert np.linalg.norm(a[s] - b[s]) <= tol * np.linalg.norm(b[s])


ODD_GRID = (16, 33, 16)
KNOBS = ("CHN_RECON_FP64", "CHN_TRANSFORMS_FP64", "CHN_SOLVE_TILE", "CHN_RECON_BUILD", "CHN_AUTOTUNE")


def odd_state(seed, laminar):
    Nx, Ny, Nz = ODD_GRID
    C = O.synthetic_state(Nx, Ny, Nz, seed=seed, laminar=laminar)
    C[1:] = 0.0
    rng = np.random.default_rng(seed)
    line = rng.standard_normal((2, 6)) * 0.1
    C[0, 0, :6, 0] += line[0]
    C[0, 1, :6, 0] += line[1]
    C[0, 1] *= 1e-10
    return C


def odd_part(C):
    return C[0, 1]


def odd_step(cc, env):
    old = {k: os.environ.pop(k, None) for k in KNOBS}
    os.environ.update({"CHN_AUTOTUNE": "0", **env})
    try:
        assert cc.c_init(*ODD_GRID, 2 * np.pi, np.pi, 2000.0, 2.0, 0.004, 1) == 0, cc.c_last_error_message()
        C, IC, AC = odd_state(1, True), odd_state(2, False), odd_state(3, False)
        AX, flow = AC.copy(), np.zeros((3, 3 * ODD_GRID[0] // 2, cc.c_qpts(), 3 * ODD_GRID[2] // 2))
        cc.c_spec2phys(C.copy(), flow)
        cc.c_primal(0, C)
        cc.c_tangent(0, 1, IC, 0)
        cc.c_adjoint(1, 0, AC, 0, 0.0)
        cc.c_adjoint_exact(1, 0, AX)
        assert cc.c_last_error() == 0, cc.c_last_error_message()
        cc.c_destroy()
        return flow[2], [odd_part(x) for x in (C, IC, AC, AX)]
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("tile,recon", [(None, None), ("16", "0"), ("8", "1"), ("8/128", "2")])
def test_a_small_spanwise_part_keeps_its_digits(tile, recon):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    env = {"CHN_SOLVE_TILE": tile, "CHN_RECON_BUILD": recon} if tile else {}
    w, tc = odd_step(cc, env)
    w0, ref = odd_step(cc, {"CHN_RECON_FP64": "1", "CHN_TRANSFORMS_FP64": "1"})
    assert np.abs(w - w0).max() <= 1e-14 * np.abs(w0).max()  # as test_gpu_recon_tc.py, of its own scale
    for a, b, tol in zip(tc, ref, PARITY):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("gi,nseg,cache", [(0, 4, "1"), (0, 4, "0"), (2, 7, "1"), (2, 7, "0"), (1, 3, "1")])
def test_concurrent_adjoint_passes_give_the_same_bits(monkeypatch, gi, nseg, cache):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    monkeypatch.setattr(V, "NSEG", nseg)
    assert 3 * V.GRIDS[gi][1] // 2 * nseg > 2 * 152
    env = {"CHN_AUTOTUNE": "0", "CHN_NO_FIELD_CACHE": "1" if cache == "0" else "0"}
    runs = [V._sweeps(cc, V.GRIDS[gi], {**env, "CHN_CONCURRENT_CHAINS": c})[0] for c in "01"]
    V._same(*runs)


@pytest.mark.parametrize("gi", [0, 1, 2])
def test_products_of_one_component_a_block_give_the_same_bits(gi):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    runs = [V._sweeps(cc, V.GRIDS[gi], {"CHN_AUTOTUNE": "0", **env})[0] for env in ({}, {"CHN_PRODUCTS_BUILD": "0"})]
    V._same(*runs)


@pytest.mark.parametrize("grid", [(144, 17, 8), (8, 17, 144)], ids=str)
def test_products_builds_of_long_transforms_give_the_same_bits(grid):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    args = (*grid, 2 * np.pi, np.pi, 2000.0, 2.0, 0.004, 2)
    runs = [V._sweeps(cc, args, {"CHN_AUTOTUNE": "0", **env})[0] for env in
            ({}, {"CHN_PRODUCTS_BUILD": "0"}, {"CHN_PRODUCTS_BUILD": "1"}, {"CHN_ADJ_PRODUCTS_PER_PASS": "3"})]
    for r in runs[1:]:
        V._same(runs[0], r)
@pytest.mark.parametrize("grids", [[(24, 17, 98), (20, 17, 12)], [(20, 17, 12), (12, 17, 14), (20, 17, 12)],
                                   [(144, 17, 8), (20, 17, 12)]], ids=str)
def test_uneven_batches(grids):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from channel import c_channel as cc
    from torch.profiler import ProfilerActivity, profile
    n = len(grids)
    i3 = lambda j: (ctypes.c_int * n)(*[g[j] for g in grids])
    d3 = lambda v: (ctypes.c_double * n)(*[v] * n)
    states = [[O.synthetic_state(*g, seed=k + i, laminar=k == 0) for i, g in enumerate(grids)] for k in (0, 10, 20)]
    C, IC, AC = (np.concatenate([x.ravel() for x in xs]) for xs in states)
    inh = (ctypes.c_int * 1)(1)
    os.environ["CHN_SWEEP_GRAPHS"] = "0"
    try:
        assert cc.lib.c_multi_init(n, i3(0), i3(1), i3(2), d3(2 * np.pi), d3(np.pi), d3(2000.0), d3(2.0), d3(0.004), 1,
                                   1, 0) == 0, cc.c_last_error_message()
        with profile(activities=[ProfilerActivity.CUDA]):
            torch.zeros(8, device="cuda").add_(1)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            assert cc.lib.c_multi_forward(0, 1, C.ctypes.data, IC.ctypes.data, inh) == 0, cc.c_last_error_message()
            assert cc.lib.c_multi_adjoint(1, 0, AC.ctypes.data, 1.0) == 0, cc.c_last_error_message()
    finally:
        os.environ.pop("CHN_SWEEP_GRAPHS", None)
        cc.lib.c_multi_destroy()
    names = {e.name for e in prof.events() if "chn::" in e.name}
    if names:
        assert any("k_phys_inverse_tc<" in k for k in names) and any("k_products_tc<" in k for k in names)
    off = 0
    for i, g in enumerate(grids):
        c, ic, ac = (states[k][i].copy() for k in range(3))
        assert cc.c_init(*g, 2 * np.pi, np.pi, 2000.0, 2.0, 0.004, 1) == 0, cc.c_last_error_message()
        cc.c_primal(0, c)
        cc.c_tangent(0, 1, ic, 1)
        cc.c_adjoint(1, 0, ac, 0, 1.0)
        assert cc.c_last_error() == 0, cc.c_last_error_message()
        cc.c_destroy()
        for a, b, tol in zip((C, IC, AC), (c, ic, ac), PARITY):
            assert np.linalg.norm(a[off:off + b.size] - b.ravel()) <= tol * np.linalg.norm(b)
        off += c.size
