// pcg_scalar.cuh -- the scalar steps of the on-chip PCG loops (included by
// pcg_cluster.cuh, inside its namespace; plain arithmetic, which a host
// compiler takes too).
//
// FP32: fp32, as the reference.  MIXED: the values of the spmv / update pair,
// which divides its double-float totals in fp64 and rounds the quotient to the
// vectors' fp32, without that division on the narrow FP64 pipe.  us per
// iteration with it and without: 24 leaves 4.53 / 3.45, 156 7.28 / 4.82 (every
// warp of the cluster divides), 1,148 7.43 / 6.49, 8,320 20.67 / 19.65.

// RN32(a / b) as fp64 gives it, for double-float totals and the set-up's fp64
// r.z (the conversions, fp64 too, stay out of the callers)
__device__ __forceinline__ double cl_wide(float2 v) { return double(v.x) + double(v.y); }
__device__ __forceinline__ double cl_wide(double v) { return v; }
template <typename A, typename B>
__device__ __noinline__ float cl_div64(A a, B b) {
  return float(cl_wide(a) / cl_wide(b));
}

// The quotient s, unless fp64 has to decide its rounding (false).  q + d is the
// quotient to about 2^-45 of it (q the leading terms' quotient, d from the
// exact remainder).  Where 2^-42 more or less does not change its rounding,
// that is the quotient's rounding and the fp64 quotient's too, and also with
// what a double-float a or b leaves of an fp64 value; where it does (once in
// some 2^17 divisions), where a remainder might underflow or something is not
// finite, it is not certain.
__device__ __forceinline__ bool cl_quot(float2 a, float2 b, float& s) {
  const float q = __fdiv_rn(a.x, b.x);
  const float w = __fmul_rn(fabsf(q), 0x1p-42f);
  const float e = __fadd_rn(__fmaf_rn(-q, b.x, a.x), __fmaf_rn(-q, b.y, a.y));
  const float d = __fmul_rn(e, __frcp_rn(b.x));  // (the reciprocal does not wait for q)
  s = __fadd_rn(q, __fadd_rn(d, w));
  const float least = fminf(fminf(fabsf(a.x), fabsf(b.x)), fabsf(q));
  return s == __fadd_rn(q, __fsub_rn(d, w)) && least > 0x1p-90f;
}
__device__ __forceinline__ bool cl_quot(float a, float b, float& s) {
  s = __fdiv_rn(a, b);
  return true;
}
// a / b, where a or b may be wide's double-float image (the r.z that the set-up
// leaves in fp64, in a segment's first iteration)
template <typename P>
__device__ __forceinline__ float cl_div(P a, P b, bool first, const double& wide, bool wide_a) {
  float s;
  if (!cl_quot(a, b, s)) {
    if (!first)
      s = cl_div64(a, b);
    else
      s = wide_a ? cl_div64(wide, b) : cl_div64(a, wide);
  }
  return s;
}

__device__ __forceinline__ void cl_split(double v, double& o) { o = v; }
__device__ __forceinline__ void cl_split(double v, float& o) { o = float(v); }
__device__ __forceinline__ void cl_split(double v, float2& o) {
  o.x = float(v);
  o.y = float(v - double(o.x));
}

// r.r <= thr of a (normalised) double-float r.r: the threshold's second part
// is rounded down, so that a second part at most that is at most the exact one
__device__ __forceinline__ void cl_threshold(double v, float2& o) {
  o.x = float(v);
  o.y = __double2float_rd(v - double(o.x));
}
__device__ __forceinline__ bool cl_at_most(float2 v, float2 thr) {
  return v.x < thr.x || (v.x == thr.x && v.y <= thr.y);
}
