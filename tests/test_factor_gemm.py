"""The CUDA-core factorization products where their tiles end.

Fronts of one pivot, of sizes next to the tile's 64 rows and columns and the
stage's 8 pivots, with and without children, one to three stages deep, of both
precisions (complex single with the CUDA cores asked for).  A panel solve is
compared with the FP64 oracle's; the bounds are those of the other panel-solve
tests, 1e-12 for complex double and 1e-4 for complex single.
"""
import math
import os

import numpy as np
import pytest

import psp_b200 as P
from conftest import oracle_for, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,cutoff", [
    (1, 1, 20, 12),    # a single point in the plane: one front
    (3, 3, 20, 1),
    (8, 8, 21, 16),    # 64 points in the plane
    (13, 5, 22, 65),   # 65, one front
    (16, 17, 19, 12),
    (21, 24, 24, 30),
])
@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
def test_panel_solves(product_lib, nx, ny, nz, cutoff, precision):
    rng = np.random.default_rng(nx + ny)
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(3, 3, 3), sigma=1.5)
    vel = rng.uniform(0.8, 1.4, (nz, ny, nx))
    B = rng.standard_normal((nz, ny, nx, 2)) + 1j * rng.standard_normal((nz, ny, nx, 2))
    O = oracle_for(disc, cutoff=cutoff)
    O.initialize(vel)
    old = os.environ.pop("PSP_B200_FACTOR_CUDA_CORES", None)
    os.environ["PSP_B200_FACTOR_CUDA_CORES"] = "1"
    try:
        H = P.DistHelmholtz(disc, cutoff=cutoff)
        H.Initialize(vel, precision=precision)
    finally:
        del os.environ["PSP_B200_FACTOR_CUDA_CORES"]
        if old is not None:
            os.environ["PSP_B200_FACTOR_CUDA_CORES"] = old
    for p in range(O.geometry().shape[0]):
        assert rel(H.solve_panel(B, p), O.solve_panel(B, p)) < (1e-12 if precision == P.FP64 else 1e-4), p
