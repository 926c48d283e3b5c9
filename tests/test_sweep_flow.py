"""Panel solves that walk the whole elimination tree in one launch.

The CUDA-core kernel (FP64, and complex single at one or two right-hand
sides) and the tensor-core kernel (complex single from three on) share an
ordered tile list.  They are compared with the FP64 oracle where a tile or
the list ends: one right-hand side, counts next to every tile width (2, 4, 8,
16, 32) and past the widest, odd counts (rows that are not 16-byte aligned),
sides that leave ragged rows and K ranges, leaves without points (cutoff 1
and 2), a tree of a single front, and columns of a wider grid.

Tolerances are those of the other sweep tests, which bound the same factors
and the same sums: 1e-12 for complex double, 1e-4 for complex single against
the oracle, and 2e-5 between the two kernels (both sum the same complex
single factors in FP32).
"""
import math
import os

import numpy as np
import pytest

import psp_b200 as P
from conftest import oracle_for, rel

pytestmark = pytest.mark.gpu

PML = 4


def _problem(nx, ny, nz, k, seed):
    rng = np.random.default_rng(seed)
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(PML,) * 3, sigma=1.5)
    vel = rng.uniform(0.8, 1.4, (nz, ny, nx))
    B = rng.standard_normal((nz, ny, nx, k)) + 1j * rng.standard_normal((nz, ny, nx, k))
    return disc, vel, np.ascontiguousarray(B)


def _handle(disc, vel, precision, cutoff, cuda_cores=False):
    old = os.environ.pop("PSP_B200_SWEEP_CUDA_CORES", None)
    try:
        if cuda_cores:
            os.environ["PSP_B200_SWEEP_CUDA_CORES"] = "1"
        H = P.DistHelmholtz(disc, cutoff=cutoff)
        H.Initialize(vel, precision=precision)  # the route is chosen here
    finally:
        os.environ.pop("PSP_B200_SWEEP_CUDA_CORES", None)
        if old is not None:
            os.environ["PSP_B200_SWEEP_CUDA_CORES"] = old
    return H


@pytest.mark.parametrize("nx,ny,nz,cutoff,ks", [
    (23, 19, 26, 12, (1, 2, 3, 4, 5, 8, 9, 16, 17, 31, 32, 33)),  # uneven, a leftover panel
    (33, 32, 21, 40, (1, 3, 16, 32)),                             # fronts next to the tile's 64 and 128 rows
    (9, 14, 24, 1, (1, 2, 3, 17)),                                # leaves without points
    (11, 8, 19, 2, (2, 7)),
    (3, 4, 20, 12, (1, 3, 20)),                                   # one front
])
def test_panel_solves_and_sweep_match_oracle(product_lib, nx, ny, nz, cutoff, ks):
    disc, vel, B = _problem(nx, ny, nz, max(ks), seed=11 + nx)
    O = oracle_for(disc, cutoff=cutoff)
    O.initialize(vel)
    H64 = _handle(disc, vel, P.FP64, cutoff)
    H32 = _handle(disc, vel, P.MIXED, cutoff)
    Hcc = _handle(disc, vel, P.MIXED, cutoff, cuda_cores=True)
    ref = O.precondition(B)
    panels = O.geometry().shape[0]
    ref_p = [O.solve_panel(B, p) for p in (0, panels - 1)]
    for k in ks:
        Bk = np.ascontiguousarray(B[..., :k])
        assert rel(H64.precondition(Bk), ref[..., :k]) < 1e-12, k
        x, c = H32.precondition(Bk), Hcc.precondition(Bk)
        assert rel(x, ref[..., :k]) < 1e-4, k
        assert rel(x, c) < 2e-5, k
        for p, r in zip((0, panels - 1), ref_p):
            assert rel(H64.solve_panel(Bk, p), r[..., :k]) < 1e-12, (k, p)
            assert rel(H32.solve_panel(Bk, p), r[..., :k]) < 1e-4, (k, p)


@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
@pytest.mark.parametrize("k", [67, 128])
def test_blocks_of_columns_of_a_wider_grid(product_lib, precision, k):
    """More than 64 right-hand sides go through the sweep in blocks of columns
    of the same grid (67: blocks of 34 and 33, starting at odd columns); every
    column is the same as on its own."""
    disc, vel, B = _problem(14, 13, 21, k, seed=5)
    H = _handle(disc, vel, precision, 12)
    x = H.precondition(B)
    for c in (0, 33, 34, k - 1):
        one = H.precondition(np.ascontiguousarray(B[..., c:c + 1]))
        assert rel(x[..., c:c + 1], one) < (1e-12 if precision == P.FP64 else 2e-5), c


def test_repeated_solves_are_identical(product_lib):
    """Which CTA takes which tile changes from run to run; the sums do not."""
    for precision, k in ((P.FP64, 5), (P.MIXED, 1), (P.MIXED, 16), (P.MIXED, 32)):
        disc, vel, B = _problem(33, 30, 22, k, seed=9)
        H = _handle(disc, vel, precision, 12)
        first = H.precondition(B)
        for _ in range(3):
            assert np.array_equal(first, H.precondition(B)), (precision, k)
