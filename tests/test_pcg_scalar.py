"""The MIXED on-chip loops' scalar steps (pcg_scalar.cuh, compiled for the host):
alpha and beta are the fp32 roundings of the fp64 quotients of the double-float
totals, as the spmv / update pair forms them, and the loop test is the fp64
comparison.  Quotients a few units of the totals' last place off a rounding
boundary, quotients anywhere, small and large ones, and what is not finite."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "fluid-sim-lb_gb300" / "csrc"

HOST = r"""
#include <cmath>
#include <cstring>
#define __device__
#define __noinline__ __attribute__((noinline))
#define __forceinline__ inline
struct float2 { float x, y; };
static inline float __fdiv_rn(float a, float b) { return a / b; }
static inline float __frcp_rn(float a) { return 1.0f / a; }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline float __double2float_rd(double v) {
  const float f = float(v);
  return double(f) > v ? nextafterf(f, -INFINITY) : f;
}
#include "pcg_scalar.cuh"
extern "C" void quotients(const float2* a, const float2* b, float* q, long n) {
  for (long i = 0; i < n; ++i) q[i] = cl_div(a[i], b[i], false, 0.0, false);
}
// fp64 numerators (wide_a) or denominators, with their double-float images
extern "C" void wide(const double* v, const float2* image, const float2* other, int wide_a,
                     float* q, long n) {
  for (long i = 0; i < n; ++i)
    q[i] = wide_a ? cl_div(image[i], other[i], true, v[i], true)
                  : cl_div(other[i], image[i], true, v[i], false);
}
extern "C" void at_most(const float2* v, const double* thr, int* r, long n) {
  for (long i = 0; i < n; ++i) {
    float2 t;
    cl_threshold(thr[i], t);
    r[i] = cl_at_most(v[i], t);
  }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pcg_scalar")
    (d / "host.cc").write_text(HOST)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    str(CSRC), "-o", str(d / "host.so"), str(d / "host.cc")], check=True)
    return ctypes.CDLL(str(d / "host.so"))


def _pair(v):
    """float64 -> normalised double-float, and the float64 that it holds."""
    hi = v.astype(np.float32)
    lo = (v - hi.astype(np.float64)).astype(np.float32)
    return np.ascontiguousarray(np.stack([hi, lo], -1)), hi.astype(np.float64) + lo


def _check(lib, a, b):
    a, av = _pair(a)
    b, bv = _pair(b)
    q = np.empty(len(a), np.float32)
    lib.quotients(a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p),
                  q.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(len(a)))
    with np.errstate(all="ignore"):
        want = (av / bv).astype(np.float32)
    same = (q == want) | (np.isnan(q) & np.isnan(want))
    assert same.all(), (a[~same][:3], b[~same][:3], q[~same][:3], want[~same][:3])


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e12, 1e-30, 1e30])
def test_quotients(lib, scale):
    rng = np.random.default_rng(1)
    n = 40000
    b = rng.uniform(1, 2, n) * 10.0 ** rng.uniform(-6, 6, n)
    _check(lib, b * rng.uniform(0.1, 10, n) * scale, b * scale)
    # near the middle of two neighbouring floats, and at both floats
    m = rng.uniform(1, 2, n).astype(np.float32).astype(np.float64)
    for half in (0.0, 0.5):
        mid = m + 2.0 ** -23 * half
        for ulps in (-8, -1, 0, 1, 8, 200):
            q = mid * 2.0 ** rng.integers(-20, 20, n)
            _check(lib, q * b * (1 + ulps * 2.0 ** -49) * scale, b * scale)


@pytest.mark.parametrize("wide_a", [True, False])
def test_first_quotients(lib, wide_a):
    """The set-up's r.z has all 53 bits; its double-float image is only what
    the certain quotients need."""
    rng = np.random.default_rng(3)
    n = 40000
    other, ov = _pair(rng.uniform(1, 2, n) * 10.0 ** rng.uniform(-6, 6, n))
    m = rng.uniform(1, 2, n).astype(np.float32).astype(np.float64) + 2.0 ** -24
    p = ctypes.c_void_p
    for ulps in (-3, -1, 0, 1, 3):
        q = m * (1 + ulps * 2.0 ** -52)
        v = np.ascontiguousarray(q * ov if wide_a else ov / q)
        image, _ = _pair(v)
        got = np.empty(n, np.float32)
        lib.wide(v.ctypes.data_as(p), image.ctypes.data_as(p), other.ctypes.data_as(p),
                 ctypes.c_int(wide_a), got.ctypes.data_as(p), ctypes.c_long(n))
        want = (v / ov if wide_a else ov / v).astype(np.float32)
        assert np.array_equal(got, want)


def test_not_finite(lib):
    a = np.array([0.0, 1.0, -1.0, np.inf, np.nan, 1.0, 1e-44, 3e38, 0.0, -5e-39, 2.0])
    b = np.array([0.0, 0.0, 0.0, 2.0, 1.0, np.nan, 1e-44, 1e-30, 3.0, 7e-40, np.inf])
    with np.errstate(all="ignore"):
        _check(lib, a, b)


def test_threshold(lib):
    rng = np.random.default_rng(2)
    n = 300000
    thr = rng.uniform(1, 2, n) * 10.0 ** rng.uniform(-12, 12, n)
    v, vv = _pair(thr * (1 + rng.integers(-20, 21, n) * 2.0 ** -50))
    r = np.empty(n, np.int32)
    lib.at_most(v.ctypes.data_as(ctypes.c_void_p), thr.ctypes.data_as(ctypes.c_void_p),
                r.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(n))
    # equality at the middle of two floats has two double-float forms
    tie = np.abs(v[:, 1].astype(np.float64)) * 2 == np.spacing(np.abs(v[:, 0])).astype(np.float64)
    assert np.array_equal(r[~tie] != 0, (vv <= thr)[~tie])
