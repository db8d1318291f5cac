"""The mixed form's reconstruction rounds a product and the sum it enters once, as the contracted
FP32 arithmetic does: PPM's limited values are the rounded 3 q - 2 r (one rounding), and each
WENO-Z substencil is within the half units of its two rounded sums (one for the last, one for the
sum before it). Built for the host with nvcc (tests/recon_host.cu)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
FP = C.POINTER(C.c_float)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("recon") / "recon_host.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", os.path.join(ROOT, "chasqui_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", so, os.path.join(HERE, "recon_host.cu")], check=True,
                   capture_output=True)
    return C.CDLL(so)


def ptr(a):
    return a.ctypes.data_as(FP)


def test_ppm_limit_rounds_once(host):
    rng = np.random.default_rng(1)
    n = 200000
    q = (1 + 0.1 * rng.normal(size=n)).astype(np.float32)
    l = (q - np.float32(0.1) * rng.random(n)).astype(np.float32)
    r = (q + np.float32(0.1) * rng.random(n)).astype(np.float32)
    l2, r2 = l.copy(), r.copy()
    host.ppm(C.c_long(n), ptr(q), ptr(l2), ptr(r2))
    q64 = q.astype(float)
    for new, old, other in ((l2, l, r), (r2, r, l)):
        cut = (new != old) & (new != q)
        assert cut.sum() > n // 10
        want = (3.0 * q64 - 2.0 * other).astype(np.float32)   # exact in FP64
        assert np.array_equal(new[cut], want[cut]), int((new != want)[cut].sum())


def test_weno_substencils_round_once_per_sum(host):
    rng = np.random.default_rng(2)
    n = 200000
    a, b, c = (rng.normal(size=n).astype(np.float32) for _ in range(3))
    out = np.empty((3, n), np.float32)
    host.weno(C.c_long(n), ptr(a), ptr(b), ptr(c), ptr(out))
    x, y, z = (v.astype(float) for v in (a, b, c))
    first = (2 * x - 7 * y, 5 * y - x, 2 * x + 5 * y)
    exact = (first[0] + 11 * z, first[1] + 2 * z, first[2] - z)
    for got, f, e in zip(out, first, exact):
        half = 0.5 * np.spacing(np.abs(f).astype(np.float32)).astype(float)
        bound = half + 0.5 * np.spacing((np.abs(e) + half).astype(np.float32))
        assert (np.abs(got - e) <= bound).all(), int((np.abs(got - e) > bound).sum())
