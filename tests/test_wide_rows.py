"""Panel solves with 32-byte accesses against the same rows without them.

Four columns of a solution, and two of the grid, are one access where rows and
pointer allow it.  A grid that starts 16 bytes past such a boundary, and column
counts that are no multiple of four or two, take the narrower ones; the sums are
the same, so the results of one column are within complex-single rounding of
each other (2e-5, as between the two sweep kernels).
"""
import math

import numpy as np
import pytest

import psp_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [4, 6, 7, 16, 24, 30, 32])
def test_grids_off_the_boundary(product_lib, k):
    import torch
    nx, ny, nz = 26, 21, 23
    rng = np.random.default_rng(k)
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(4, 4, 4), sigma=1.5)
    H = P.DistHelmholtz(disc)
    H.Initialize(rng.uniform(0.8, 1.4, (nz, ny, nx)), precision=P.MIXED)
    n = nx * ny * nz * k
    rhs = torch.randn(n, dtype=torch.complex128, device="cuda")
    out = []
    for offset in (0, 1, 2):
        store = torch.empty(n + 2, dtype=torch.complex128, device="cuda")
        B = store[offset:offset + n]
        B.copy_(rhs)
        H.precondition_device(B)
        out.append(B.clone())
    assert torch.linalg.norm(out[1] - out[0]) < 2e-5 * torch.linalg.norm(out[0])
    assert torch.equal(out[2], out[0])
    one = rhs.view(-1, k)[:, k - 1].contiguous()
    H.precondition_device(one)
    assert torch.linalg.norm(out[1].view(-1, k)[:, k - 1] - one) < 2e-5 * torch.linalg.norm(one)
