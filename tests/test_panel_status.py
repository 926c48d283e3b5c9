"""A panel solve that could not be carried out says so.

Panels that are factored when a solve reaches them report a zero or non-finite
pivot in a status word, and so do the solve's own bounded waits.  Every entry
point that solves panels reads it before it returns; none hands back a grid that
was not solved as a success.
"""
import math
import os

import numpy as np
import pytest

import psp_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
def test_bad_pivot_of_a_recomputed_panel(product_lib, precision):
    nx, ny, nz = 9, 8, 22
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(3, 3, 3), sigma=1.5)
    old = os.environ.get("PSP_B200_RESIDENT_PANELS")
    os.environ["PSP_B200_RESIDENT_PANELS"] = "0"  # Initialize factors nothing
    try:
        H = P.DistHelmholtz(disc)
        B = np.ones((nz, ny, nx, 2), dtype=np.complex128)
        vel = np.ones((nz, ny, nx))
        H.Initialize(vel, precision=precision)
        H.solve_panel(B, 1)
        vel[nz // 2] = np.nan
        H.Initialize(vel, precision=precision)
        bad = [p for p, (v, depth, _, _) in enumerate(H.geometry())
               if v <= nz - 1 - nz // 2 < v + depth]
        with pytest.raises(P.PspRuntimeError, match="pivot"):
            H.solve_panel(B, bad[0])
        with pytest.raises(P.PspRuntimeError, match="pivot"):
            H.precondition(B)
        vel[:] = 1
        H.Initialize(vel, precision=precision)
        assert np.isfinite(H.solve_panel(B, bad[0])).all()
    finally:
        del os.environ["PSP_B200_RESIDENT_PANELS"]
        if old is not None:
            os.environ["PSP_B200_RESIDENT_PANELS"] = old
