"""A panel solve whose wait runs out.

The kernels that walk the elimination tree bound every wait.  When one runs out
(here on a counter that nothing sets) they report it in the status word, and
what later launches start from, the ticket, the fronts' counters and the
arrivals of split tiles, is at zero again: a count left behind made the next
solve on the same plan sum partial tiles that were not written yet.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def driver(product_lib, tmp_path_factory):
    out = str(tmp_path_factory.mktemp("drv") / "flow_timeout")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    libdir = os.path.join(ROOT, "psp_b200")
    cxx = ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []
    subprocess.run([nvcc] + cxx + ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                                   "--expt-relaxed-constexpr", "-I", os.path.join(libdir, "csrc"),
                                   os.path.join(ROOT, "tests", "drivers", "flow_timeout.cu"), "-o", out,
                                   "-L", libdir, "-lpsp_b200", "-Xlinker", "-rpath", "-Xlinker", libdir], check=True)
    return out


def test_driver_compiles(driver):
    assert os.path.exists(driver)


@pytest.mark.gpu
def test_counters_are_at_zero_after_a_wait_ran_out(driver):
    r = subprocess.run([driver], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
