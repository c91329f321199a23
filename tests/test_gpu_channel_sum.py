"""The mixed form's adjoint channel sums against exact sums of the same FP32 rows
(math.fsum), beside an FP64 sum in the order that one warp takes (lanes over the
channels, then the lanes' sums in pairs): over rows whose values spread over 0,
12 and 36 bits, with and without cancellation, of as many channels as a lane's
first and second rounds, a block of them and two sensors have.

The fixed-point sum rounds every value at most once, within 2^-59 of the largest
value's leading bit, and the result once: its rms error over the rows may be no
larger than the FP64 sum's, plus the result's own rounding."""
import ctypes as ct
import math
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    from crtmv3_gb300 import build
    so = str(tmp_path_factory.mktemp("sum") / "sum.so")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-shared", "-I" + build.CSRC, "-o", so,
                                                        os.path.join(ROOT, "tests", "harness", "sum_harness.cu")],
                   check=True, cwd=ROOT)
    return ct.CDLL(so)


def _device(lib, x):
    out = np.full(x.shape[0], np.nan)
    assert lib.run_channel_sum(x.ctypes.data_as(ct.c_void_p), ct.c_longlong(x.shape[0]), x.shape[1],
                               out.ctypes.data_as(ct.c_void_p)) == 0
    return out


def _warp_fp64(x):
    n, L = x.shape
    y = np.zeros((n, (L + 31) // 32 * 32))
    y[:, :L] = x
    lanes = np.zeros((n, 32))
    for c in range(y.shape[1] // 32):
        lanes = lanes + y[:, 32 * c:32 * c + 32]
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, np.arange(32) ^ o]
    return lanes[:, 0]


@pytest.mark.parametrize("L", [1, 31, 33, 511, 513, 616, 2211, 9000])
@pytest.mark.parametrize("bits", [0, 12, 36])
@pytest.mark.parametrize("cancel", [False, True])
def test_sum_no_less_exact_than_fp64(lib, L, bits, cancel):
    rng = np.random.default_rng([L, bits, cancel])
    n = 400
    x = (rng.uniform(1.0, 2.0, (n, L)) * rng.choice([-1.0, 1.0], (n, L) if cancel else (n, 1)) *
         2.0 ** -rng.uniform(0.0, bits, (n, L)) * 10.0 ** rng.integers(-20, 20, (n, 1))).astype(np.float32)
    exact = [math.fsum(r) for r in x.astype(np.float64)]
    top = np.abs(x).max(axis=1).astype(np.float64)
    rms = lambda s: math.sqrt(np.mean([((a - e) / m) ** 2 for a, e, m in zip(s, exact, top)]))  # noqa: E731
    final = 2.0 ** -53 * math.sqrt(np.mean((np.array(exact) / top) ** 2))
    assert rms(_device(lib, x)) <= rms(_warp_fp64(x.astype(np.float64))) + final


def test_rows_without_a_fixed_point(lib):
    """Rows of zeros and subnormals, and infinities and NaNs, as FP64 adds them."""
    tiny = np.float32(1e-45)
    x = np.zeros((6, 70), np.float32)
    x[1, 3], x[1, 69] = tiny, -3 * tiny
    x[2, 5] = np.inf
    x[3, 5], x[3, 6] = np.inf, -np.inf
    x[4, 7] = np.nan
    x[5] = 1.0
    x[5, 0] = tiny
    got = _device(lib, x)
    assert got[0] == 0.0 and got[1] == -2.0 * float(tiny) and got[2] == np.inf and np.isnan(got[3]) and np.isnan(got[4])
    assert got[5] == 69.0
