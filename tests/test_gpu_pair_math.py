"""The exponential and the reciprocal square root of the pair kernels
(sf_pairs.cuh) against extended precision (80-bit) over the ranges that the
kernels meet, in the stated error bounds.

expScaled, FP64: 2^(c s / 64), u = 2^-53.  Relative error: table entry u, the
last fused multiply-add u, series of 2^(f/64) - 1 (at most 0.0055) 3.5e-17 by
truncation and 4 roundings of its value, f itself half a rounding of 1/2 in
units of ln 2 / 64: below 2.5 u, down to 2^-1000.  The form for Gaussians that
underflow has the same bits there; below 2^-1021 its result only has to be
between 0 and 2^-1020.  FP32: ex2.approx 2^-22, the rounding of the product
c s 2^-24 |c s| ln 2 and those of c and s themselves (exact here), down to
2^-126, then 0.  invSqrt: seed within 2^-20, one third-order step: 5/16 e^3 <
1e-17 with e <= 2^-19, the residual's rounding 0.75 u and the last one u:
below 3 u; FP32: rsqrtf, 2 units in the last place."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    so = str(tmp_path_factory.mktemp("pair_math") / "pair_math.so")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(ROOT, "n2p2_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "pair_math.cu"),
                    "-o", so], check=True)
    lib = ctypes.CDLL(so)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    tab = np.exp2(np.arange(64, dtype=np.longdouble) / 64).astype(np.float64)

    def call(s, c):
        s, c = (np.ascontiguousarray(x, dtype=np.float64) for x in (s, c))
        out = [np.empty(s.size, dtype=t) for t in (np.float64, np.float64, np.float64, np.float32, np.float32)]
        assert lib.run(s.size, p(s), p(c), p(tab), *[p(x) for x in out]) == 0
        return out
    return call


def _arguments():
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(0.0, 1.0, 20000), rng.uniform(0.0, 64.0, 20000), rng.uniform(0.0, 64 * 1000.0, 40000),
                        np.arange(0, 64 * 1000, 0.5)[:60000],            # table boundaries, ties of the rounding
                        np.arange(1, 4000) * (1 + 2.0 ** -40), 2.0 ** -np.arange(1.0, 60.0), [0.0, 1e-300]])
    s = rng.uniform(0.01, 400.0, x.size)
    s[-2:] = 0.0, 1e-300
    return s, -np.where(s > 0, x / np.where(s > 0, s, 1.0), 3.0)


def test_exponential_fp64(run):
    s, c = _arguments()
    got, wide = run(s, c)[:2]
    want = np.exp2(s.astype(np.longdouble) * c.astype(np.longdouble) / 64)
    err = np.abs((got - want) / want).astype(np.float64)
    assert err.max() <= 2.5 * U
    assert np.array_equal(got, wide)


def test_exponential_fp64_underflow(run):
    x = np.concatenate([np.linspace(1000.0, 1100.0, 5001), np.geomspace(1100.0, 2.0 ** 24, 4000)])   # powers of 1/2
    s = np.full(x.size, 3.0)
    c = -64 * x / 3.0
    got = run(s, c)[1]
    with np.errstate(under="ignore"):
        want = np.exp2(s.astype(np.longdouble) * c.astype(np.longdouble) / 64)
    assert np.all((got >= 0.0) & (got <= np.maximum(2.0 ** -1020, 2 * want)))
    normal = x < 1020.0
    assert (np.abs(got[normal] - want[normal]) / want[normal]).max() <= 2.5 * U


def test_exponential_fp32(run):
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(0.0, 1.0, 20000), rng.uniform(0.0, 125.0, 20000)])
    s = rng.uniform(0.01, 400.0, x.size).astype(np.float32).astype(np.float64)
    c = -(x / s).astype(np.float32).astype(np.float64)
    got = run(s, c)[3].astype(np.float64)
    want = np.exp2((s * c).astype(np.longdouble)).astype(np.float64)
    assert np.all(np.abs(got - want) <= want * (2.0 ** -22 + 2.0 ** -24 * (1.0 + np.abs(s * c) * np.log(2.0))))
    far = np.geomspace(150.0, 2.0 ** 24, 1000)
    assert np.all(run(np.full(far.size, 1.0), -far)[3] == 0.0)


def test_reciprocal_root(run):
    rng = np.random.default_rng(3)
    s = np.concatenate([rng.uniform(0.1, 600.0, 100000), np.geomspace(1e-12, 1e12, 100001), 2.0 ** np.arange(-40.0, 40.0),
                        2.0 ** np.arange(-40.0, 40.0) * (1 + 2.0 ** -52), 2.0 ** np.arange(-40.0, 40.0) * (1 - 2.0 ** -53)])
    out = run(s, np.zeros(s.size))
    want = 1.0 / np.sqrt(s.astype(np.longdouble))
    assert (np.abs(out[2] - want) / want).max() <= 3 * U
    s32 = s.astype(np.float32).astype(np.longdouble)
    want = 1.0 / np.sqrt(s32)
    assert (np.abs(out[4] - want) / want).max() <= 2 * 2.0 ** -23
