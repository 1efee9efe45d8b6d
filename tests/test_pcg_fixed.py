"""The fixed-point words of the resident loop's grid barriers (pcg_fixed.cuh,
compiled for the host): the sum of 152 CTAs' partials, taken as the barrier takes
it, against exact arithmetic.  The units are 2^-40 of the previous total, and
the wider types carry 2^-40 of those in a second word, so a total that keeps at
least 2^33 units is off by its rounding and 152 cuts at most."""
import ctypes
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "fluid-sim-lb_gb300" / "csrc"

HOST = r"""
#include <cmath>
#include <cstring>
#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
static inline float2 make_float2(float x, float y) { return float2{x, y}; }
template <typename A, typename B> static inline A bits(B v) { A a; memcpy(&a, &v, sizeof(a)); return a; }
static inline unsigned __float_as_uint(float v) { return bits<unsigned>(v); }
static inline long long __double_as_longlong(double v) { return bits<long long>(v); }
static inline double __longlong_as_double(long long v) { return bits<double>(v); }
static inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
static inline float __ll2float_rn(long long v) { return float(v); }
static inline long long __float2ll_rn(float v) { return llrintf(v); }
#include "pcg_fixed.cuh"

// One barrier's sum of n partials at the scale of `like`; 0 when the words hold
// it, 1 when a partial is out of range, 2 when the total is too small
template <typename P, bool TWO, bool LANES>
static int total(const P* v, int n, P like, P* out) {
  const int s = res_scale(like);
  long long hi = 0, lo = 0;
  for (int i = 0; i < n; i += LANES ? 32 : 1) {
    long long h[32], l[32];
    for (int j = 0; j < (LANES ? 32 : 1); ++j)
      if (!res_fix(v[i + j], s, h[j], l[j])) return 1;
    if (LANES) {  // a warp's limbs
      unsigned sum[4] = {0, 0, 0, 0};
      for (int j = 0; j < 32; ++j) {
        int q[4];
        res_limbs(h[j], l[j], q);
        for (int k = 0; k < 4; ++k) sum[k] += unsigned(q[k]);
      }
      const int q[4] = {int(sum[0]), int(sum[1]), int(sum[2]), int(sum[3])};
      res_unlimb(q, h[0], l[0]);
    }
    hi += h[0];
    lo += TWO ? l[0] : 0;
  }
  if (hi < (1ll << 33)) return 2;
  res_unfix(hi, lo, s, *out);
  return 0;
}
extern "C" int total_f(const float* v, int n, float like, float* o) { return total<float, false, false>(v, n, like, o); }
extern "C" int total_f2(const float2* v, int n, const float2* like, float2* o) { return total<float2, true, false>(v, n, *like, o); }
extern "C" int total_d(const double* v, int n, double like, double* o) { return total<double, true, true>(v, n, like, o); }
"""
P = ctypes.c_void_p


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pcg_fixed")
    (d / "host.cc").write_text(HOST)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    str(CSRC), "-o", str(d / "host.so"), str(d / "host.cc")], check=True)
    return ctypes.CDLL(str(d / "host.so"))


def _run(lib, kind, v, like):
    """(code, total as a Fraction) and the exact sum."""
    n = len(v)
    if kind == "f":
        v = v.astype(np.float32)
        o = ctypes.c_float()
        code = lib.total_f(v.ctypes.data_as(P), n, ctypes.c_float(like), ctypes.byref(o))
        return code, Fraction(o.value), sum(map(Fraction, map(float, v)))
    if kind == "d":
        o = ctypes.c_double()
        code = lib.total_d(v.ctypes.data_as(P), n, ctypes.c_double(like), ctypes.byref(o))
        return code, Fraction(o.value), sum(map(Fraction, map(float, v)))
    hi = v.astype(np.float32)
    lo = (v - hi.astype(np.float64)).astype(np.float32)
    pair = np.ascontiguousarray(np.stack([hi, lo], -1))
    lk = np.array([like, 0.0], np.float32)
    o = np.zeros(2, np.float32)
    code = lib.total_f2(pair.ctypes.data_as(P), n, lk.ctypes.data_as(P), o.ctypes.data_as(P))
    exact = sum(Fraction(float(a)) + Fraction(float(b)) for a, b in pair)
    return code, Fraction(float(o[0])) + Fraction(float(o[1])), exact


# rounding of the total: half a unit of its last place (the double-float form
# holds 48 bits), and a cut of one unit per partial, of 2^-40 (2^-33 at worst)
# of the total for FP32 and 2^-40 of that for the wider types
BARS = {"f": 2.0 ** -24, "f2": 2.0 ** -48, "d": 2.0 ** -53}


@pytest.mark.parametrize("kind", ["f", "f2", "d"])
@pytest.mark.parametrize("signs", [False, True])
def test_totals(lib, kind, signs):
    rng = np.random.default_rng(4)
    top = {"f": 30, "f2": 25, "d": 900}[kind]
    n = 152 * (32 if kind == "d" else 1)
    taken = 0
    for _ in range(300):
        v = rng.uniform(0, 1, n) * 10.0 ** rng.uniform(-4, 0, n)
        if signs:
            v *= rng.choice([-1, 1], n, p=[0.3, 0.7])
        v *= 2.0 ** rng.integers(-top, top)
        like = float(abs(v.sum()) * 2.0 ** rng.uniform(-5, 6.5))  # the previous total
        code, got, exact = _run(lib, kind, v, like)
        if code:
            continue
        taken += 1
        cut = n * 2.0 ** (-33 if kind == "f" else -73)
        assert abs(got - exact) <= (BARS[kind] + cut) * exact, (v, like)
    assert taken > 250


@pytest.mark.parametrize("kind", ["f", "f2", "d"])
def test_out_of_range(lib, kind):
    """Totals far below the previous one, partials far above it and what is
    not finite go to the sums through memory."""
    n = 152 * (32 if kind == "d" else 1)
    v = np.full(n, 1.0 / n)
    assert _run(lib, kind, v, 1.0)[0] == 0
    assert _run(lib, kind, v * 2.0 ** -8, 1.0)[0] == 2
    assert _run(lib, kind, -v, 1.0)[0] == 2
    assert _run(lib, kind, 0 * v, 1.0)[0] == 2
    for bad in (2.0 ** 6.5, -2.0 ** 6.5, np.inf, -np.inf, np.nan):
        w = v.copy()
        w[7] = bad
        with np.errstate(invalid="ignore"):
            code = {"f": lambda: lib.total_f(w.astype(np.float32).ctypes.data_as(P), n,
                                             ctypes.c_float(1.0), ctypes.byref(ctypes.c_float())),
                    "d": lambda: lib.total_d(w.ctypes.data_as(P), n, ctypes.c_double(1.0),
                                             ctypes.byref(ctypes.c_double())),
                    "f2": lambda: lib.total_f2(
                        np.ascontiguousarray(np.stack([w, 0 * v], -1).astype(np.float32)
                                             ).ctypes.data_as(P), n,
                        np.array([1.0, 0.0], np.float32).ctypes.data_as(P),
                        np.zeros(2, np.float32).ctypes.data_as(P))}[kind]()
        assert code == 1, bad
