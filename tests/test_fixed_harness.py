"""The layer solver for known angle counts (scatter_fixed.cuh) against the
run-time form, on the CPU: the same FP32 operations in the same order, so the
same bits (compiled without contraction into fused multiply-adds), over its
angle counts and thin, ordinary, thick and nearly conservative layers."""
import ctypes as ct
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fixed") / "fixed.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "crtmv3_gb300", "csrc"), "-o", so,
                    os.path.join(ROOT, "tests", "harness", "fixed_harness.cpp")], check=True, cwd=ROOT)
    lib = ct.CDLL(so)
    lib.run_layers.restype = ct.c_long
    lib.run_layers.argtypes = [ct.c_int, ct.c_int, ct.c_double, ct.c_double, ct.c_double]
    return lib


@pytest.mark.parametrize("NS", [2, 3, 4])
@pytest.mark.parametrize("tau_lo,tau_hi,w_hi", [(1e-12, 1e-8, 1.0), (1e-6, 10.0, 0.999), (10.0, 300.0, 0.9999999)])
def test_fixed_equals_runtime(lib, NS, tau_lo, tau_hi, w_hi):
    assert lib.run_layers(NS, 500, tau_lo, tau_hi, w_hi) == 0
