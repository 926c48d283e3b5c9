"""GMRES's column reductions (norms, dots) against the FP64 operator.

One launch forms the block sums and adds them, so the sizes are those where a
launch ends: a grid that fits one block, several blocks with a remainder, more
points than one pass of every block (the unrolled loop and its tail), one
column, odd and many columns, and more columns than a block has threads to
spare (one point per block).

The residual that GMRES reports after its last step is max_r |b - A x| / |b|
from device norms.  Recomputed with the NumPy operator from the returned x it
can differ by the rounding of b - A x, about 27 terms of size |A| |x| at 1.1e-16:
|A| |x| / |b| stays below 1e3 on these grids, so 1e-11 bounds it.  Each column's
dots are checked by the number of steps: with the FP64 preconditioner a block
needs as many as its slowest column does alone (all columns of the small blocks,
a sample of the wide ones).
"""
import math

import numpy as np
import pytest

import psp_b200 as P
from conftest import oracle_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,k", [
    (5, 5, 18, 1),      # one block
    (9, 8, 18, 3),      # a few blocks, the last one short
    (9, 8, 18, 67),
    (9, 8, 18, 300),     # one point per block
    (40, 37, 30, 16),    # every block takes more than one pass, and a remainder
])
def test_norms_and_dots(product_lib, nx, ny, nz, k):
    rng = np.random.default_rng(nx + k)
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(3, 3, 3), sigma=1.5)
    vel = rng.uniform(0.8, 1.4, (nz, ny, nx))
    B = rng.standard_normal((nz, ny, nx, k)) + 1j * rng.standard_normal((nz, ny, nx, k))
    B *= 10.0 ** np.arange(k) ** 0.3  # columns of different sizes
    O = oracle_for(disc)
    O.form_operator(vel)
    H = P.DistHelmholtz(disc)
    H.Initialize(vel, precision=P.FP64)
    X = B.copy()
    H.Solve(X, 10, 1e-6)
    last = H.last_stats
    res = np.linalg.norm((B - O.multiply(X)).reshape(-1, k), axis=0) / np.linalg.norm(B.reshape(-1, k), axis=0)
    assert res.max() < 1e-6
    assert abs(last["final_max_rel_resid"] - res.max()) < 1e-11
    steps = []
    for r in range(k) if k < 20 else (0, k // 2, k - 1):
        H.Solve(np.ascontiguousarray(B[..., r:r + 1]), 10, 1e-6)
        steps.append(H.last_stats["iterations"])
    assert max(steps) == last["iterations"] if k < 20 else max(steps) <= last["iterations"]
