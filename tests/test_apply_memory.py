"""What multiply_device keeps between calls takes no room from other calls.

The temporary of B := A B stays with the handle, up to 1 GiB.  On a device that is
nearly full a later Solve has to go in the same blocks of right-hand sides as
without it, and to find the memory for them; and after Finalize nothing is kept.
"""
import math

import numpy as np
import pytest

import psp_b200 as P

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def test_multiply_does_not_narrow_a_later_solve(product_lib):
    import torch
    nx, ny, nz, k = 60, 60, 300, 64  # the temporary is 1.0 GiB
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(3, 3, 3), sigma=1.5)
    H = P.DistHelmholtz(disc)
    H.Initialize(np.ones((nz, ny, nx)), precision=P.MIXED)
    n = nx * ny * nz
    B = torch.randn(n * k, dtype=torch.complex128, device="cuda")
    hog = None
    try:
        free = torch.cuda.mem_get_info()[0]
        hog = torch.empty(free - 4 * GIB, dtype=torch.uint8, device="cuda")
        width = H.solve_block_width(10 ** 6)  # (so many that blocks are as wide as they can be)
        H.multiply_device(B)
        assert H.solve_block_width(10 ** 6) == width
        H.set_max_iterations(1)  # the memory is the point, not the solution
        X = B[:n * min(width, k)]
        H.Solve(X, 20, 1e-12)
        H.multiply_device(B)
    finally:
        del hog
        torch.cuda.empty_cache()
        H.Finalize()
    free = torch.cuda.mem_get_info()[0]
    H.multiply_device(B)
    assert torch.cuda.mem_get_info()[0] == free
