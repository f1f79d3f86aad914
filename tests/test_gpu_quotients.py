"""The kernels' reciprocals and quotients (csrc/quotient.cuh) against IEEE
division over the ranges they state and at the ends of FP32's.

Bound: one unit in the last place of the correctly rounded value.  recip: the
approximation's error of 2^-23 squared is below 2^-45, then one rounding; quot
and quot_d: the first quotient is within 2^-22, its remainder exact, the
correction's error below 2^-44, then one rounding."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tooling_gb300", "csrc")
SOURCE = """
#include "quotient.cuh"
__global__ void k(int op, int n, const double* a, const double* b, float* o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x = (float)a[i], d = (float)b[i];
  o[i] = op == 0 ? recip(d) : op == 1 ? quot(x, d, recip(d)) : op == 2 ? quot(x, d, 1.f / d) : quot_d(a[i], b[i]);
}
extern "C" int run(int op, int n, const double* a, const double* b, float* o) {
  double *da, *db;
  float* d;
  if (cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&d, n * 4)) return 1;
  cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(op, n, da, db, d);
  const int e = cudaMemcpy(o, d, n * 4, cudaMemcpyDeviceToHost);
  cudaFree(da); cudaFree(db); cudaFree(d);
  return e;
}
"""
RECIP, QUOT_RECIP, QUOT, QUOT_D = range(4)
N = 1 << 20


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cu").write_text(SOURCE)
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, str(d / "q.cu"), "-o", str(d / "q.so")],
                   check=True)
    f = ctypes.CDLL(str(d / "q.so")).run

    def call(op, a, b):
        a, b = (np.ascontiguousarray(x, np.float64) for x in np.broadcast_arrays(a, b))
        o = np.empty(a.size, np.float32)
        assert f(op, a.size, a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p),
                 o.ctypes.data_as(ctypes.c_void_p)) == 0
        return o
    return call


def _near(got, want):
    """Equal, or neighbours among the FP32 numbers of one sign."""
    g, w = got.view(np.int32).astype(np.int64), want.view(np.int32).astype(np.int64)
    return (got == want) | ((np.sign(got) == np.sign(want)) & (np.abs(g - w) <= 1))


def _floats(rng, n, lo, hi):
    x = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n)).astype(np.float32)
    x[: n // 8] = np.ldexp(1.0, rng.integers(lo, hi, n // 8))  # powers of two, and their neighbours
    x[n // 8: n // 4] = np.nextafter(x[: n // 4 - n // 8], np.float32(np.inf))
    return x


def test_reciprocals(run):
    rng = np.random.default_rng(1)
    x = _floats(rng, N, -126, 126)
    assert _near(run(RECIP, 1, x), np.float32(1) / x).all()
    first, last = np.float32(2.0 ** -126), np.float32(2.0 ** 126)
    ends = np.float32([first, -first, last, -last])
    assert _near(run(RECIP, 1, ends), np.float32(1) / ends).all()
    assert (run(RECIP, 1, np.float32([np.nextafter(last, np.float32(np.inf)), 2.0 ** 127, 3.4028235e38])) == 0).all()  # past the range
    assert np.isnan(run(RECIP, 1, np.float32([0, 1e-40, np.inf, np.nan]))).all()


@pytest.mark.parametrize("op", [QUOT_RECIP, QUOT])
def test_quotients(run, op):
    rng = np.random.default_rng(2)
    d = _floats(rng, N, -126, 126)
    n = _floats(rng, N, -100, 126) * rng.choice(np.float32([-1, 1]), N)
    rng.shuffle(n)
    with np.errstate(over="ignore", under="ignore"):
        want = n / d
    ok = (np.abs(want) > 2.0 ** -125) & (np.abs(want) < 2.0 ** 126)
    assert ok.sum() > N // 4 and _near(run(op, n[ok], d[ok]), want[ok]).all()
    e = d[d > 2.0 ** -100]
    assert (run(op, e, e) == 1).all()


def test_quotients_of_doubles(run):
    rng = np.random.default_rng(3)
    a = np.ldexp(rng.uniform(1, 2, N), rng.integers(-170, 170, N)) * rng.choice([-1.0, 1.0], N)
    b = np.ldexp(rng.uniform(1, 2, N), rng.integers(-170, 170, N))
    with np.errstate(over="ignore", under="ignore"):
        want = (a / b).astype(np.float32)
    assert _near(run(QUOT_D, a, b), want).all()
    assert (run(QUOT_D, np.float64([0.0, 1e300, -1e300, 1e39]), np.float64([2.0, 1e-300, 1e-300, 1e25])) ==
            np.float32([0, np.inf, -np.inf, 1e14])).all()
