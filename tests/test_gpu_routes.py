"""Calls whose kernels a rule picks, against the kernels of another rule.

Long transforms (144x17x8, 8x17x200): planes that fit one block, whose tables'
rows have no room in the sums kept between two stages, run the split
tensor-core passes and agree with the FP64 kernels to rounding.  The oracle built with
and without FMA contraction differs by at most (primal, tangent, adjoint)
3.3e-13, 4.0e-13, 3.4e-13 there; the one-step parity tolerances 5e-12, 1e-11,
3e-11 hold.
"""
import numpy as np
import pytest

from conftest import has_gpu
from test_gpu_builds import _step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(144, 17, 8, 1, 2), (8, 17, 200, 1, 2)], ids=lambda c: "x".join(map(str, c)))
def test_long_transforms_match_the_fp64_kernels(case):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from channel import c_channel as cc
    for a, b, tol in zip(_step(cc, *case, False), _step(cc, *case, True), (5e-12, 1e-11, 3e-11, 3e-11)):
        for s in range(a.shape[0]):
            assert np.linalg.norm(a[s] - b[s]) <= tol * np.linalg.norm(b[s])
