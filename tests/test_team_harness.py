"""The adding's inverse by a team of lanes (scatter_team_math.cuh) on an emulated
warp, against the per-thread function: the same FP32 or FP64 operations in the
same order, so the same bits (compiled without contraction into fused
multiply-adds on both sides), over the angle classes, matrix sizes, weak and
strong coupling, mixed sizes within a warp and partly filled warps."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def team(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("team") / "team.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "crtmv3_gb300", "csrc"), "-o", so,
                    os.path.join(ROOT, "tests", "harness", "team_harness.cpp")], check=True, cwd=ROOT)
    lib = ct.CDLL(so)
    lib.run_inverse.restype = ct.c_long
    return lib


INPUT = np.dtype([("n", "i4"), ("m", "f4", 100)])
SIZES = {4: (2, 3, 4), 5: (5,), 6: (6,), 10: (9, 10)}


@pytest.mark.parametrize("NZ", [4, 5, 6, 10])
def test_team_inverse_equals_thread(team, NZ):
    assert team.input_bytes() == INPUT.itemsize
    rng = np.random.default_rng(NZ)
    for trial in range(60):
        teams = int(rng.integers(1, team.teams_per_warp(NZ) + 1))
        y = np.zeros(teams, INPUT)
        y["n"] = rng.choice(SIZES[NZ], size=teams)
        # weak coupling is eliminated in FP32, strong in FP64
        y["m"] = rng.normal(size=(teams, 100)) * rng.choice([0.01, 0.1], size=teams)[:, None]
        assert team.run_inverse(NZ, y.ctypes.data_as(ct.c_void_p), teams) == 0, trial
