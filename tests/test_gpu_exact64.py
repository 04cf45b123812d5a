"""The FP64 building blocks of csrc/fv_exact64.cuh against IEEE arithmetic.

Sums and products as three-register fused operations, quotients and square
roots from FP32 seeds with a rounding test: every result must be the IEEE one,
bit for bit (the tolerance is none).  The operands cover random significands
and exponents, exact and nearly exact results, quotients closest to a midpoint
of two doubles, powers of two and their neighbours, zeros, infinities, NaN,
subnormals and the edges of the fast path's ranges.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from fv3d_gb300 import build as fvbuild

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fv_exact64.cuh"
using namespace fv;
__global__ void ops(int n, const double* a, const double* b, double* add, double* sub, double* mul, double* quo,
                    double* sq) {
  opaque64_init();
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const X64 x = a[i], y = b[i];
    add[i] = (x + y).v;
    sub[i] = (x - y).v;
    mul[i] = (x * y).v;
    quo[i] = div64(x, y).v;
    sq[i] = sqrt64(x).v;
  }
}
extern "C" int run(int n, const double* a, const double* b, double* out) {
  double* d = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  if (cudaMalloc(&d, 7 * bytes) != cudaSuccess) return 1;
  cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
  ops<<<608, 256>>>(n, d, d + n, d + 2 * n, d + 3 * n, d + 4 * n, d + 5 * n, d + 6 * n);
  const cudaError_t e = cudaMemcpy(out, d + 2 * n, 5 * bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact64")
    src, so = str(d / "ops.cu"), str(d / "ops.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call([fvbuild._nvcc(), "-fmad=false", *fvbuild.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                           "-I", fvbuild.CSRC, "-I", fvbuild.INCLUDE, "-shared", "-o", so, src])
    assert os.path.exists(so)
    return ctypes.CDLL(so)


def check(lib, a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    out = np.empty((5, a.size))
    dp = ctypes.POINTER(ctypes.c_double)
    assert lib.run(a.size, *(x.ctypes.data_as(dp) for x in (a, b, out))) == 0
    with np.errstate(all="ignore"):
        want = [a + b, a - b, a * b, a / b, np.sqrt(a)]
    for name, got, ref in zip(("a + b", "a - b", "a * b", "a / b", "sqrt(a)"), out, want):
        same = (got.view(np.int64) == ref.view(np.int64)) | (np.isnan(got) & np.isnan(ref))
        bad = np.flatnonzero(~same)
        assert bad.size == 0, (name, bad.size, a[bad[:3]].tolist(), b[bad[:3]].tolist(), got[bad[:3]].tolist(),
                               ref[bad[:3]].tolist())


def significands(rng, n):
    return 1.0 + rng.integers(0, 1 << 52, n) * 2.0 ** -52


@pytest.mark.parametrize("span", [0, 3, 60, 150, 400, 800, 1020])
def test_random_operands(lib, span):
    rng = np.random.default_rng(span)
    n = 1 << 22
    a = np.ldexp(significands(rng, n), rng.integers(-span, span + 1, n)) * rng.choice([1.0, 1.0, 1.0, -1.0], n)
    b = np.ldexp(significands(rng, n), rng.integers(-span, span + 1, n)) * rng.choice([1.0, 1.0, -1.0], n)
    check(lib, a, b)


def test_exact_and_nearly_exact_results(lib):
    """Quotients and roots that are representable, and one unit beside them."""
    rng = np.random.default_rng(1)
    n = 1 << 20
    q = np.ldexp(rng.integers(1, 1 << 26, n).astype(np.float64), rng.integers(-30, 30, n))
    b = np.ldexp(rng.integers(1, 1 << 26, n).astype(np.float64), rng.integers(-30, 30, n))
    for a in (q * b, np.nextafter(q * b, np.inf), np.nextafter(q * b, 0.0), q * q):
        check(lib, a, b)
    check(lib, np.nextafter(q * q, np.inf), q)
    near = 1.0 + rng.integers(-8, 9, n) * 2.0 ** -52  # beside powers of two
    check(lib, np.ldexp(near, rng.integers(-20, 20, n)), np.ldexp(1.0 + rng.integers(-8, 9, n) * 2.0 ** -52,
                                                                 rng.integers(-20, 20, n)))


def test_quotients_beside_midpoints(lib):
    """a / b as close to a midpoint of two doubles as it can be: for an odd
    53-bit b, m = -1/b mod 2^54 is a midpoint's numerator (54 bits) and
    a = (b m + 1) / 2^54 an integer, so a / b = m / 2^54 + 1 / (b 2^54)."""
    rng = np.random.default_rng(2)
    a, b = [], []
    for x in rng.integers(1 << 52, 1 << 53, 20000):
        x = int(x) | 1
        for sign in (1, -1):
            m = (-sign * pow(x, -1, 1 << 54)) % (1 << 54)
            v = (x * m + sign) >> 54
            if m >> 53 and v < 1 << 53:
                a.append(float(v))
                b.append(float(x))
    assert len(a) > 5000
    a, b = np.array(a), np.array(b)
    check(lib, a, b)
    check(lib, -np.ldexp(a, -60), np.ldexp(b, -40))


def test_roots_beside_midpoints(lib):
    """x = RN((g + half a unit)^2): roots within a quarter of a unit of a midpoint, both parities."""
    rng = np.random.default_rng(3)
    g = significands(rng, 1 << 21)
    hi = g * g + g * 2.0 ** -52
    for x in (hi, np.nextafter(hi, np.inf), np.nextafter(hi, 0.0), 2.0 * hi):
        check(lib, x, g)


def test_special_operands(lib):
    v = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** -1021, 1.5,
                  2.0, 3.0, 4.0, 1.7976931348623157e308, 0.1, 1.0 / 3.0, np.nextafter(1.0, 2.0), np.nextafter(1.0, 0.0),
                  np.nextafter(2.0, 0.0), np.nextafter(4.0, 0.0), 1.4, -0.1])
    edges = np.array([-750, -700, -150, 150, 700, 800], dtype=np.float64)  # of the fast path's ranges
    edges = np.concatenate([2.0 ** edges, np.nextafter(2.0 ** edges, 0), 1.7 * 2.0 ** edges])
    v = np.concatenate([v, edges, -edges])
    a, b = np.meshgrid(v, v)
    check(lib, a.ravel(), b.ravel())
