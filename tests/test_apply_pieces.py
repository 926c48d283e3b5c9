"""The operator's rows in pieces.

A block of the operator kernels takes 128 points of a row, or what is left of it; a
launch of few blocks takes the rows in equal pieces, of up to 32 points when these
are very few or long.  Every entry is formed by the
same arithmetic whatever its piece, so a wide block of columns equals its columns
alone bit for bit, on rows next to the pieces' lengths, for whole grids, slabs of
planes and the residual, on either side of the rule (half a wave of blocks, four
waves, 24 columns).  The oracle bounds one column as in the other operator
tests: 27 terms of complex double, 1e-13.
"""
import math

import numpy as np
import pytest

import psp_b200 as P
from conftest import oracle_for, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,k", [
    (31, 3, 18, 5), (33, 2, 18, 24), (65, 4, 18, 23), (96, 5, 18, 24), (127, 4, 19, 64),
    (129, 3, 18, 33), (257, 2, 18, 16),
    (129, 30, 20, 23), (129, 30, 20, 24),   # more than half a wave, less than four
    (130, 60, 44, 24),                      # more than four
])
def test_wide_blocks_equal_their_columns(product_lib, nx, ny, nz, k):
    import torch
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(3, 3, 3), sigma=1.5)
    vel = np.random.default_rng(nx).uniform(0.8, 1.4, (nz, ny, nx))
    H = P.DistHelmholtz(disc)
    H.Initialize(vel, precision=P.MIXED)
    stream = torch.cuda.ExternalStream(H.stream_ptr())
    torch.manual_seed(k)
    n = nx * ny * nz
    X = torch.randn(n, k, dtype=torch.complex128, device="cuda")
    R = torch.randn(n, k, dtype=torch.complex128, device="cuda")

    def calls(x, r):
        kk = x.shape[1]
        x, r = x.contiguous(), r.contiguous()
        y, s, d = (torch.zeros_like(x) for _ in range(3))
        z = x.clone()
        stream.wait_stream(torch.cuda.current_stream())  # the handle works on a stream of its own
        H.multiply_slab(x.view(-1), y.view(-1), kk, 0, nz, 0)
        H.multiply_slab(x.view(-1), d.view(-1), kk, 0, nz, 0, r.view(-1))
        H.multiply_slab(x.view(-1), s.view(-1), kk, 3, 2, 0)
        H.multiply_device(z.view(-1))
        return y, d, s, z

    wide = calls(X, R)
    assert torch.equal(wide[0], wide[3])
    assert torch.equal(wide[0].view(nz, -1)[3:5], wide[2].view(nz, -1)[3:5])
    for c in (0, k // 2, k - 1):
        for a, b in zip(wide, calls(X[:, c:c + 1], R[:, c:c + 1])):
            assert torch.equal(a[:, c:c + 1], b), c
    O = oracle_for(disc)
    O.form_operator(vel)
    x = X[:, k - 1].cpu().numpy().reshape(nz, ny, nx, 1)
    assert rel(wide[0][:, k - 1].cpu().numpy().reshape(x.shape), O.multiply(x)) < 1e-13
