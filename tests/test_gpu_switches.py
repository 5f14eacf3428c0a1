"""The switches that ask for a kernel's build hold for small launches too.

A launch of few blocks has builds of its own (a component or field per block,
4-column tiles).  CHN_FIXED_SIZES has to keep the builds compiled for a grid's
sizes in or out there as well; CHN_PRODUCTS_BUILD, CHN_ADJ_PRODUCTS_PER_PASS, CHN_SOLVE_TILE
and CHN_RECON_BUILD ask for a build of the others and get it.  The kernels that
ran are read by name from the CUDA activity record.

So are those that a rule on sizes picks: the inverse of planes of few kx columns
(8x17x128) runs the FFTs in batches, the split tensor-core passes where planes are few.
"""
import ctypes
import os
import re

import numpy as np
import pytest

import oracle as O
from conftest import has_gpu

pytestmark = pytest.mark.gpu

KNOBS = ("CHN_SOLVE_TILE", "CHN_FIXED_SIZES", "CHN_ADJ_PRODUCTS_PER_PASS", "CHN_RECON_BUILD", "CHN_PRODUCTS_BUILD",
         "CHN_AUTOTUNE", "CHN_SWEEP_GRAPHS")
GRIDS = [(32, 65, 32), (16, 33, 16)]


def kernels(grid, env, nseg=1):
    """names of the kernels of one step each way of a small batch"""
    from channel import c_channel as cc
    from torch.profiler import ProfilerActivity, profile
    old = {k: os.environ.pop(k, None) for k in KNOBS}
    os.environ.update({"CHN_AUTOTUNE": "0", "CHN_SWEEP_GRAPHS": "0", **env})
    try:
        assert cc.c_init(*grid, 2 * np.pi, np.pi, 2000.0, 2.0, 0.004, 1) == 0, cc.c_last_error_message()
        lib = cc.lib
        assert lib.c_batch_init(nseg, 1, 0) == 0, cc.c_last_error_message()
        C, IC, AC = (np.stack([O.synthetic_state(*grid, seed=k + s, laminar=k == 0) for s in range(nseg)])
                     for k in (0, 10, 20))
        AX, inh = AC.copy(), (ctypes.c_int * 1)(1)
        try:
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                assert lib.c_batch_forward(0, 1, C.ctypes.data, IC.ctypes.data, inh) == 0, cc.c_last_error_message()
                assert lib.c_batch_adjoint(1, 0, AC.ctypes.data, 1.0) == 0, cc.c_last_error_message()
                assert lib.c_batch_adjoint_exact(1, 0, AX.ctypes.data) == 0, cc.c_last_error_message()
        finally:
            lib.c_batch_destroy()
        cc.c_destroy()
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v
    names = {e.name for e in prof.events() if "chn::" in e.name}
    if not names:
        pytest.skip("no kernel activity record on this machine")
    return names


def of(names, kernel):
    got = [n for n in names if re.search(rf"\b{kernel}\b", n)]
    assert got, (kernel, sorted(names))
    return got


@pytest.fixture(scope="module", autouse=True)
def gpu():
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]):  # the process's first record can come back empty
        torch.zeros(8, device="cuda").add_(1)
        torch.cuda.synchronize()


@pytest.mark.parametrize("grid", GRIDS, ids=str)
def test_fixed_sizes(grid):
    run_time, compiled = (kernels(grid, {"CHN_FIXED_SIZES": v}) for v in "01")
    for k in ("k_recon_few", "k_solve", "k_solve_T", "k_products_tc"):
        assert not any("SizesCT" in n for n in of(run_time, k))
        assert all("SizesCT" in n for n in of(compiled, k))


@pytest.mark.parametrize("grid", GRIDS, ids=str)
@pytest.mark.parametrize("env", [{"CHN_PRODUCTS_BUILD": "0"}, {"CHN_PRODUCTS_BUILD": "1"},
                                 {"CHN_ADJ_PRODUCTS_PER_PASS": "1"}, {"CHN_ADJ_PRODUCTS_PER_PASS": "3"}], ids=str)
def test_products(grid, env):
    assert of(kernels(grid, {}), "k_assemble")  # components in blocks of their own by default
    names = kernels(grid, env)
    assert not any("k_assemble" in n for n in names)
    planes = {int(re.search(r"k_products_tc<[^,]*, (\d)", n).group(1)) for n in of(names, "k_products_tc")}
    want = {"CHN_PRODUCTS_BUILD": {"0": {1, 3}, "1": {2}}, "CHN_ADJ_PRODUCTS_PER_PASS": {"1": {1}, "3": {1, 3}}}
    (switch, value), = env.items()
    assert planes == want[switch][value]


@pytest.mark.parametrize("env,gone", [({"CHN_SOLVE_TILE": "16"}, r"k_solve(_T)?<[^>]*>?, 4,"),
                                      ({"CHN_RECON_BUILD": "0"}, "k_recon_few")], ids=str)
def test_tiles(env, gone):
    assert any(re.search(gone, n) for n in kernels(GRIDS[1], {}))
    assert not any(re.search(gone, n) for n in kernels(GRIDS[1], env))


@pytest.mark.parametrize("grid,nseg,kernel", [((8, 17, 128), 1, "k_z_inv_tc"), ((8, 17, 128), 8, "k_phys_inverse"),
                                              ((20, 17, 108), 20, "k_z_inv_tc")], ids=str)
def test_inverse_of_narrow_planes(grid, nseg, kernel):
    names = kernels(grid, {}, nseg)
    inverse = {k for k in ("k_z_inv_tc", "k_phys_inverse", "k_phys_inverse_tc", "k_tz_inv")
               if any(re.search(rf"\b{k}\b", n) for n in names)}
    assert inverse == {kernel}
