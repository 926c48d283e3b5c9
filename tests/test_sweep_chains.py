"""Routes and accumulation chains of complex-single panel solves.

The tensor core truncates as it accumulates, so a tile keeps at most three stages
(48 complex K) in one accumulator; its chains are summed in FP32.  K-chunks of 32
columns are one chain each, summed across tiles; chunks of 64 are a chain of three
stages and one of one; chunks of 512 hold up to eleven chains, summed inside the tile;
unset, the tiling rule chooses.  All of them, and the CUDA-core kernel, sum the same
products in FP32, so they agree to the bound between the kernels in the other sweep
tests, 2e-5 (a lost or repeated chain is off by O(1)), and with the FP64 oracle
to 1e-4.  The root fronts have K ranges of several hundred columns.
"""
import os

import pytest

import psp_b200 as P
from conftest import oracle_for, rel
from psp_b200 import workloads as W

pytestmark = pytest.mark.gpu

ROUTES = {
    "rule": {},
    "one chain a tile": {"PSP_B200_SWEEP_TC_CHUNK": "32"},
    "two chains a tile": {"PSP_B200_SWEEP_TC_CHUNK": "64"},
    "long tiles": {"PSP_B200_SWEEP_TC_CHUNK": "512"},
    "bounded": {"PSP_B200_SWEEP_TC_MAX_CHUNK": "128"},
    "CUDA cores": {"PSP_B200_SWEEP_CUDA_CORES": "1"},
}
SWITCHES = ("PSP_B200_SWEEP_TC_CHUNK", "PSP_B200_SWEEP_TC_MAX_CHUNK", "PSP_B200_SWEEP_CUDA_CORES")


@pytest.mark.parametrize("k", [3, 16, 32])
def test_every_route_gives_the_same_solves(product_lib, k):
    w = W.small_case(interior=(40, 36, 12), pml=5, freq=2.5, k=k, seed=21, top_pml=True)
    O = oracle_for(w.disc)
    O.initialize(w.velocity)
    panels = range(O.geometry().shape[0])
    ref, ref_p = O.precondition(w.rhs), [O.solve_panel(w.rhs, p) for p in panels]
    old = {s: os.environ.pop(s, None) for s in SWITCHES}
    out, out_p = {}, {}
    try:
        for name, env in ROUTES.items():
            os.environ.update(env)
            H = P.DistHelmholtz(w.disc)
            H.Initialize(w.velocity, precision=P.MIXED)
            out[name] = H.precondition(w.rhs)  # the switches are read up to the first panel solve
            for s in env:
                del os.environ[s]
            out_p[name] = [H.solve_panel(w.rhs, p) for p in panels]
            H.Finalize()
    finally:
        for s, v in old.items():
            os.environ.pop(s, None)
            if v is not None:
                os.environ[s] = v
    for name in ROUTES:
        assert rel(out[name], ref) < 1e-4, name
        assert rel(out[name], out["CUDA cores"]) < 2e-5, name
        assert rel(out[name], out["rule"]) < 2e-5, name
        for p in panels:
            assert rel(out_p[name][p], ref_p[p]) < 1e-4, (name, p)
            assert rel(out_p[name][p], out_p["CUDA cores"][p]) < 2e-5, (name, p)
