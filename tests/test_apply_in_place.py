"""B := A B through the memory that a handle keeps between calls.

The sizes are those where the route changes: a row next to a block's 128
points, a single step and its copy, and a grid of more than 1 GiB, which goes in
slabs of planes.  Against the oracle the operator is 27 terms of
complex double per entry, so 1e-13 bounds the relative difference; the slabs
and the calls of several threads do the same arithmetic, bit for bit.
"""
import math
import threading

import numpy as np
import pytest

import psp_b200 as P
from conftest import oracle_for, rel

pytestmark = pytest.mark.gpu


def _handle(nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    h = 1.0 / 24
    disc = P.Discretization(2 * math.pi * 0.8 / (10 * h), nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h,
                            pml=(3, 3, 3), sigma=1.5)
    vel = rng.uniform(0.8, 1.4, (nz, ny, nx))
    H = P.DistHelmholtz(disc)
    H.Initialize(vel, precision=P.MIXED)
    return disc, vel, H


@pytest.mark.parametrize("nx,ny,nz", [(5, 5, 18), (127, 3, 18), (128, 2, 19), (130, 3, 18)])
def test_rows_and_columns(product_lib, nx, ny, nz):
    disc, vel, H = _handle(nx, ny, nz, nx)
    O = oracle_for(disc)
    O.form_operator(vel)
    rng = np.random.default_rng(1)
    for k in (1, 3, 16, 5):  # (the kept memory grows, and is larger than needed)
        B = rng.standard_normal((nz, ny, nx, k)) + 1j * rng.standard_normal((nz, ny, nx, k))
        assert rel(H.multiply(B), O.multiply(B)) < 1e-13, k


def test_slabs_of_planes(product_lib):
    import torch
    nx, ny, nz, k = 60, 60, 300, 64  # 1.1 GB
    _, _, H = _handle(nx, ny, nz, 2)
    B = torch.randn(nz * ny * nx, k, dtype=torch.complex128, device="cuda")
    cols = [B[:, c:c + 16].contiguous() for c in (0, 16, 32, 48)]
    H.multiply_device(B.view(-1))
    for c, part in enumerate(cols):
        H.multiply_device(part.view(-1))
        assert torch.equal(B[:, 16 * c:16 * c + 16], part), c


def test_threads_share_the_memory(product_lib):
    import torch
    nx, ny, nz = 40, 30, 20
    _, _, H = _handle(nx, ny, nz, 3)
    ks = (1, 8, 3, 16)
    inputs = [torch.randn(nz * ny * nx * k, dtype=torch.complex128, device="cuda") for k in ks]
    want = [x.clone() for x in inputs]
    for x in want:
        for _ in range(3):
            H.multiply_device(x)
    torch.cuda.synchronize()
    for x in inputs:  # all at once, on one handle
        x.got = x.clone()
    torch.cuda.synchronize()

    def work(x):
        for _ in range(3):
            H.multiply_device(x.got)

    threads = [threading.Thread(target=work, args=(x,)) for x in inputs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, w in zip(inputs, want):
        assert torch.equal(x.got, w)
