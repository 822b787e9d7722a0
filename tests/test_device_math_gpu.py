"""The reciprocals, quotients and square roots that the 3D stage kernels use,
compiled from the kernels' own headers into a small library.  1/rho in float is
the IEEE quotient: every mantissa, and zeros, infinities and subnormals.  The
branch-free double forms are compared with extended precision.  Their errors
in units of the last place (relative 2^-53 is half of one to one unit):
  rcp_nb         the series' remainder e^3 (2^-60) and one rounding: 0.51
  div_nb         the remainder of the quotient corrects it: 0.5
  over_sqrt_nb   s = num y and the last sum round once each, the rounding of a y
                 enters e and half of it the result: 2.5 at most (measured 1.43;
                 with num = a 0.76)"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from batsrus_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "bx_stage_unit.cuh"
using namespace bx;
__global__ void kd(int op, const double *a, const double *b, double *o, long n) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
    const double x = a[q], y = b[q];
    o[q] = op == 0 ? rcp_nb(x) : op == 1 ? div_nb(x, y) : op == 2 ? over_sqrt_nb(x, y) : op == 3 ? sqrt_nb(x)
         : op == 4 ? sqrt0_nb(x) : fast_speed(x, y, 0.0, 2.0);
  }
}
__global__ void kf(const float *a, float *o, long n) {
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x)
    o[q] = rcp_cell(a[q]);
}
template <class F> static int with(const void *a, const void *b, void *o, size_t bytes, F f) {
  void *d[3] = {};
  int r = 0;
  for (auto &p : d) r |= cudaMalloc(&p, bytes);
  if (!r) {
    r |= cudaMemcpy(d[0], a, bytes, cudaMemcpyHostToDevice);
    r |= cudaMemcpy(d[1], b, bytes, cudaMemcpyHostToDevice);
    if (!r) f(d[0], d[1], d[2]);
    r |= cudaGetLastError();
    r |= cudaMemcpy(o, d[2], bytes, cudaMemcpyDeviceToHost);
  }
  for (auto p : d) cudaFree(p);
  return r;
}
extern "C" int run_d(int op, const double *a, const double *b, double *o, long n) {
  return with(a, b, o, 8 * n, [&](void *x, void *y, void *z) {
    kd<<<592, 256>>>(op, (const double *)x, (const double *)y, (double *)z, n); });
}
extern "C" int run_f(const float *a, float *o, long n) {
  return with(a, a, o, 4 * n, [&](void *x, void *, void *z) { kf<<<592, 256>>>((const float *)x, (float *)z, n); });
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    (d / "m.cu").write_text(SOURCE)
    cmd = [build.NVCC] + build.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
                                       "-I", build.CSRC, "-shared", "-o", str(d / "m.so"), str(d / "m.cu"), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(os.path.join(str(d), "m.so"))


def device(lib, op, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = np.ascontiguousarray(a if b is None else b, dtype=np.float64)
    o = np.empty_like(a)
    p = ctypes.c_void_p
    assert lib.run_d(op, p(a.ctypes.data), p(b.ctypes.data), p(o.ctypes.data), ctypes.c_long(a.size)) == 0
    return o


def numbers(rng, n, lo, hi):
    """random mantissas and powers of two, and mantissas next to 1 and 2"""
    m = 1.0 + rng.random(n)
    m[: n // 8] = 1.0 + rng.integers(0, 64, n // 8) * 2.0 ** -52
    m[n // 8: n // 4] = 2.0 - rng.integers(1, 64, n // 4 - n // 8) * 2.0 ** -52
    return np.ldexp(m, rng.integers(lo, hi, n))


def ulps(got, exact):
    return float(np.max(np.abs(got.astype(np.longdouble) - exact) / np.spacing(np.abs(exact.astype(np.float64)))))


def test_float_reciprocal_is_the_ieee_quotient(lib):
    one = np.arange(1 << 23, dtype=np.uint32)
    x = np.concatenate([(one | np.uint32(e << 23)).view(np.float32) for e in (127, 64, 190)] +
                       [np.array([0.0, -0.0, np.inf, -np.inf, 1e-45, 1e-39, 3e38, -0.7], dtype=np.float32)])
    o = np.empty_like(x)
    p = ctypes.c_void_p
    assert lib.run_f(p(x.ctypes.data), p(o.ctypes.data), ctypes.c_long(x.size)) == 0
    with np.errstate(divide="ignore", over="ignore"):
        ref = np.float32(1.0) / x
    assert np.array_equal(o.view(np.uint32), ref.view(np.uint32)), int((o.view(np.uint32) != ref.view(np.uint32)).sum())


@pytest.mark.parametrize("op,name,bound", [(0, "rcp_nb", 0.51), (1, "div_nb", 0.5), (2, "over_sqrt_nb", 2.5),
                                           (3, "sqrt_nb", 2.5)])
def test_double_forms_against_extended_precision(lib, op, name, bound):
    """2^20 random operands and as many with mantissas next to 1 and 2; exponents
    up to 2^900 for the one-operand forms, 2^60 (the range of a quotient of
    speeds, densities and pressures in SI units is less) for the others"""
    rng = np.random.default_rng(11)
    e = 900 if op in (0, 3) else 60
    a, b = numbers(rng, 1 << 21, -e, e), numbers(rng, 1 << 21, -e, e)
    A, B = a.astype(np.longdouble), b.astype(np.longdouble)
    exact = [1 / A, A / B, A / np.sqrt(B), np.sqrt(A)][op]
    got = device(lib, op, a, b)
    assert ulps(got, exact) <= bound, (name, ulps(got, exact))
    if op == 1:
        assert np.array_equal(got, a / b)  # corrected by its remainder: the IEEE quotient


def test_double_forms_at_the_ends_of_their_ranges(lib):
    """the smallest and largest operands that still give numbers, and the two
    roots that are taken of zeros: sqrt0_nb adds 1e-290, fast_speed 1e-280 under
    its inner root and 1e-290 under the outer one"""
    a = np.array([1e-307, 1e-300, 1e-200, 1e200, 1e300, 4e307])
    assert np.allclose(device(lib, 0, a), 1 / a, rtol=2.5e-16, atol=0)
    assert np.allclose(device(lib, 3, a), np.sqrt(a), rtol=5e-16, atol=0)
    assert np.allclose(device(lib, 4, [0.0]), 1e-145, rtol=1e-15, atol=0)
    # fast_speed(gamma p, B^2, 0, 2 rho = 2): sqrt(gamma p + B^2) down to the
    # clamp, where it is sqrt((G + 1e-140) / 2)
    gp, b2 = np.array([0.0, 0.0, 1e-100, 1e-30, 1e140]), np.array([0.0, 1e-30, 1e-100, 1e-12, 1e100])
    assert np.allclose(device(lib, 5, gp, b2), np.sqrt((gp + b2 + np.maximum(gp + b2, 1e-140)) / 2), rtol=1e-15, atol=0)
