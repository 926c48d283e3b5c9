"""Column tiles of the CUDA-core panel solves.

More than 16 right-hand sides go in tiles of 16 columns, or of 32 on grids whose
wide levels outweigh the chain of levels and when the tiles of 16 are even in
number.  Either way the columns' sums are the same up to the order of the K
splits, so a wide block agrees with its columns taken 16 at a time to the bounds of
the other sweep tests: 1e-12 for complex double, 2e-5 for complex single.  Both
sides of the rule, its remainders, and columns of a wider grid.
"""
import math
import os

import numpy as np
import pytest

import psp_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,ks", [
    (30, 28, 21, (17, 31, 33, 64)),      # tiles of 16
    (170, 164, 18, (17, 32, 33, 49, 64, 96)),  # of 32 (k = 33: of 16, 96: two blocks of 48)
])
@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
def test_wide_blocks_equal_narrow_ones(product_lib, precision, nx, ny, nz, ks):
    import torch
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(4, 4, 4), sigma=1.5)
    vel = np.random.default_rng(3).uniform(0.8, 1.4, (nz, ny, nx))
    old = os.environ.pop("PSP_B200_SWEEP_CUDA_CORES", None)
    os.environ["PSP_B200_SWEEP_CUDA_CORES"] = "1"
    try:
        H = P.DistHelmholtz(disc)
        H.Initialize(vel, precision=precision)
    finally:
        del os.environ["PSP_B200_SWEEP_CUDA_CORES"]
        if old is not None:
            os.environ["PSP_B200_SWEEP_CUDA_CORES"] = old
    torch.manual_seed(nx)
    rhs = torch.randn(nx * ny * nz, max(ks), dtype=torch.complex128, device="cuda")
    want = torch.empty_like(rhs)
    stream = torch.cuda.ExternalStream(H.stream_ptr())

    def precondition(x):
        stream.wait_stream(torch.cuda.current_stream())  # the handle works on a stream of its own
        H.precondition_device(x.view(-1))
        return x

    for c in range(0, max(ks), 16):
        want[:, c:c + 16] = precondition(rhs[:, c:c + 16].contiguous())
    for k in ks:
        x = precondition(rhs[:, :k].contiguous())
        err = torch.linalg.norm(x - want[:, :k]) / torch.linalg.norm(want[:, :k])
        assert err < (1e-12 if precision == P.FP64 else 2e-5), k
