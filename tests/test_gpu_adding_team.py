"""The mixed form's adding and its adjoint by teams of lanes (adding_team_kernel)
against the per-thread kernel in FP32 on the same layer records: the same bits,
over every angle count, scattering and clear layers side by side in a warp,
weak and strong coupling (FP32 and FP64 inverses), layers that failed, profiles
without clouds and stream counts that do not exist, at channel counts around a
warp's and a CTA's teams.  What a record does not hold is filled with NaN."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    from crtmv3_gb300 import build
    so = str(tmp_path_factory.mktemp("adding") / "adding.so")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-shared", "-I" + build.CSRC, "-o", so,
                                                        os.path.join(ROOT, "tests", "harness", "adding_harness.cu")],
                   check=True, cwd=ROOT)
    lib = ct.CDLL(so)
    lib.gauss_angle.restype = ct.c_double
    return lib


def _inputs(lib, NC, L, seed):
    rng = np.random.default_rng(seed)
    streams = (2, 4, 6) if NC == 5 else (8, 16)
    P, K = 9, 14
    ns = rng.choice(streams, P).astype(np.int32)
    ns[:len(streams)] = streams
    ns[-1] = 5 if NC == 5 else 12              # no such stream set
    nc = np.ones(P, np.int32)
    nc[-2] = 0                                 # clear
    nl = rng.integers(2, K + 1, P).astype(np.int32)
    mu = rng.uniform(0.4, 1.0, P)
    nS = (ns + 2) // 2
    for p in range(0, P - 1, 2):               # the sensor's angle one of the quadrature's
        mu[p] = lib.gauss_angle(int(nS[p]), int(rng.integers(0, nS[p])))
    NE = 2 + 2 * NC * NC + NC
    rec = np.full((P, K, NE, L), np.nan, np.float32)
    for p in range(P - 1):
        n = int(nS[p]) + (p % 2)
        kind = rng.choice([0.0, 1.0], (K, L), p=[0.4, 0.6]).astype(np.float32)
        od = rng.uniform(0.0, 1.5, (K, L))
        ref = rng.choice([0.02, 0.3, 0.9], (K, 1, 1, L))
        cosines = rng.uniform(0.2, 1.0, n)
        T = np.exp(-od[:, None] / cosines[None, :, None])[:, :, None] * np.eye(n)[None, :, :, None]
        T = T * 0.7 + rng.uniform(0.0, 0.2 / n, (K, n, n, L))
        R = rng.uniform(0.0, 2.0 / n, (K, n, n, L)) * ref
        s = kind == 1.0
        for i in range(n):
            for j in range(n):
                rec[p, :, 2 + i * NC + j] = np.where(s, T[:, i, j], np.nan)
                rec[p, :, 2 + NC * NC + i * NC + j] = np.where(s, R[:, i, j], np.nan)
            rec[p, :, 2 + 2 * NC * NC + i] = np.where(s, rng.uniform(1.0, 60.0, (K, L)), np.nan)
        if p in (3, 4):                        # a few pairs with a layer that failed
            kind[rng.integers(0, nl[p]), rng.choice(L, max(1, L // 5), replace=False)] = -5.0
        rec[p, :, 0], rec[p, :, 1] = kind, od
    cover = rng.choice([-1.0, 0.4, 1.0], P)
    spec = np.stack([rng.uniform(50.0, 150.0, L), rng.uniform(900.0, 1500.0, L), rng.uniform(0.0, 0.1, L),
                     rng.uniform(0.999, 1.0, L), rng.uniform(1e-4, 1e-2, L), rng.uniform(700.0, 1000.0, L)])
    return dict(P=P, K=K, NE=NE, ints=np.concatenate([nl, nc, ns]).astype(np.int32),
                prof=np.concatenate([mu, rng.uniform(270.0, 300.0, P), cover]), spec=spec,
                temperature=rng.uniform(200.0, 300.0, (P, K)), emissivity=rng.uniform(0.3, 1.0, (P, L)), rec=rec,
                tau=rng.uniform(0.0, 0.3, (P, K, L)).astype(np.float32))


def _run(lib, teams, NC, L, x):
    P, K = x["P"], x["K"]
    o = dict(lba=np.full((P, K, x["NE"], L), -777.0, np.float32), cb=np.full((P, 4, L), -777.0),
             status=np.zeros(P, np.int32), nfs=np.full((P, L), -7, np.int32), error=np.zeros(1, np.int32))
    a = [np.ascontiguousarray(x[f]) for f in ("ints", "prof", "spec", "temperature", "emissivity", "rec", "tau")]
    rc = lib.run_adding(int(teams), NC, P, L, K, *[v.ctypes.data_as(ct.c_void_p) for v in a],
                        *[o[f].ctypes.data_as(ct.c_void_p) for f in ("lba", "cb", "status", "nfs", "error")])
    assert rc == 0
    return o


@pytest.mark.parametrize("NC,L", [(5, 1), (5, 7), (5, 33), (5, 130), (10, 1), (10, 3), (10, 17), (10, 65)])
def test_teams_give_the_threads_bits(lib, NC, L):
    x = _inputs(lib, NC, L, [NC, L])
    t, r = _run(lib, True, NC, L, x), _run(lib, False, NC, L, x)
    nl = x["ints"][:x["P"]]
    assert np.array_equal(t["nfs"], r["nfs"]) and np.array_equal(t["status"], r["status"])
    assert (t["error"] != 0) == (r["error"] != 0)
    assert (r["status"][[3, 4, x["P"] - 1]] == 16).all() and np.isfinite(r["cb"]).all()
    assert t["cb"].tobytes() == r["cb"].tobytes()
    failed = 0
    for p in range(x["P"]):
        for l in range(L):
            a, b = t["lba"][p, :, :, l], r["lba"][p, :, :, l]
            if b[0, 0] == -1.0:                # a failed pair: its kinds alone are read
                failed += 1
                assert (a[:nl[p], 0] == -1.0).all() and (b[:nl[p], 0] == -1.0).all(), (p, l)
            else:
                assert a.tobytes() == b.tobytes(), (p, l, np.argwhere(a != b)[:4])
    assert failed > L
