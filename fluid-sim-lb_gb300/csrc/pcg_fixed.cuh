// pcg_fixed.cuh -- the fixed-point words of the resident loop's grid barriers
// (included by pcg_resident.cuh, inside its namespace; integer arithmetic,
// which a host compiler takes too).  A value v at scale s is hi + lo 2^-40 in
// units of 2^-s.

// mant 2^sh (mant < 2^53) as hi + lo 2^-40, cut towards zero; false when out
// of range
__device__ __forceinline__ bool res_fix(unsigned long long mant, int sh, bool neg, long long& hi,
                                        long long& lo) {
  lo = 0;
  if (sh >= 0) {
    if (mant != 0ull && (sh > 46 || (mant >> (46 - sh)) != 0ull)) return false;
    hi = static_cast<long long>(sh > 46 ? 0ull : mant << sh);
  } else {
    const int r = -sh;
    const unsigned long long h = r < 64 ? mant >> r : 0ull;
    if (h >> 46) return false;
    hi = static_cast<long long>(h);
    const unsigned long long rest = r < 64 ? mant - (h << r) : mant;  // below 2^r
    lo = static_cast<long long>(r <= 40 ? rest << (40 - r) : (r - 40 < 64 ? rest >> (r - 40) : 0ull));
  }
  if (neg) {
    hi = -hi;
    lo = -lo;
  }
  return true;
}
// v 2^s
__device__ __forceinline__ bool res_fix(float v, int s, long long& hi, long long& lo) {
  const unsigned u = __float_as_uint(v);
  const int e = int((u >> 23) & 255u);
  const unsigned m = (u & 0x7FFFFFu) | (e ? 0x800000u : 0u);
  return res_fix(static_cast<unsigned long long>(m), (e ? e : 1) - 150 + s, (u >> 31) != 0u, hi, lo) &&
         e != 255;
}
__device__ __forceinline__ bool res_fix(double v, int s, long long& hi, long long& lo) {
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  const int e = int((u >> 52) & 2047ull);
  const unsigned long long m = (u & 0xFFFFFFFFFFFFFull) | (e ? 0x10000000000000ull : 0ull);
  return res_fix(m, (e ? e : 1) - 1075 + s, (u >> 63) != 0ull, hi, lo) && e != 2047;
}
__device__ __forceinline__ bool res_fix(float2 v, int s, long long& hi, long long& lo) {
  long long h, l;
  const bool a = res_fix(v.x, s, hi, lo), b = res_fix(v.y, s, h, l);
  hi += h;
  lo += l;
  return a && b;
}
// FP64 sums are integers all the way from the lanes: the FP64 pipe takes 64
// cycles for one warp's addition, where a limb of 26 bits is summed over a
// warp by one instruction (12.0 against 8.1 us per iteration at one leaf per
// SM; for MIXED, whose lanes add double-float pairs, the same measured slower,
// 8.65 against 8.07 us at 3 leaves per SM).  X = hi 2^40 + lo in four limbs
// (the last one signed), and back from limb sums.
__device__ __forceinline__ void res_limbs(long long hi, long long lo, int (&l)[4]) {
  constexpr unsigned long long kM = (1ull << 26) - 1ull;
  const unsigned long long xl = static_cast<unsigned long long>(hi) << 40;
  const unsigned long long t = xl + static_cast<unsigned long long>(lo);
  const long long xh = (hi >> 24) + (lo >> 63) + (t < xl ? 1 : 0);
  l[0] = int(t & kM);
  l[1] = int((t >> 26) & kM);
  l[2] = int(((t >> 52) | (static_cast<unsigned long long>(xh) << 12)) & kM);
  l[3] = int(xh >> 14);
}
__device__ __forceinline__ void res_unlimb(const int (&l)[4], long long& hi, long long& lo) {
  constexpr long long kM = (1ll << 26) - 1ll;
  long long c = l[0];
  const long long l0 = c & kM;
  c = (c >> 26) + l[1];
  const long long l1 = c & kM;
  c = (c >> 26) + l[2];
  const long long l2 = c & kM;
  const long long l3 = (c >> 26) + l[3];
  lo = l0 + ((l1 & 0x3FFFll) << 26);
  hi = (l1 >> 14) + (l2 << 12) + (l3 << 38);
}
// (hi + lo 2^-40) 2^-s of a total (hi >= 2^33, 0 <= lo): for the wider types
// the leading 64 bits t, t 2^-k of the units, rounded
__device__ __forceinline__ unsigned long long res_lead64(long long hi, long long lo, int& k) {
  const unsigned long long y = static_cast<unsigned long long>(hi + (lo >> 40));
  k = __clzll(static_cast<long long>(y));
  return (y << k) | ((static_cast<unsigned long long>(lo) & ((1ull << 40) - 1ull)) >> (40 - k));
}
__device__ __forceinline__ void res_unfix(long long hi, long long, int s, float& v) {
  v = scalbnf(__ll2float_rn(hi), -s);
}
__device__ __forceinline__ void res_unfix(long long hi, long long lo, int s, double& v) {
  int k;
  const unsigned long long t = res_lead64(hi, lo, k);
  const unsigned long long m = (t >> 11) + ((t >> 10) & 1ull);  // 53 bits (2^53 carries over)
  v = __longlong_as_double(static_cast<long long>(
      (static_cast<unsigned long long>(1086 - k - s) << 52) + (m - (1ull << 52))));
}
__device__ __forceinline__ void res_unfix(long long hi, long long lo, int s, float2& v) {
  int k;
  const long long t = static_cast<long long>(res_lead64(hi, lo, k) >> 1);
  const float h = __ll2float_rn(t);
  const float l = __ll2float_rn(t - __float2ll_rn(h));
  v = make_float2(scalbnf(h, 1 - k - s), scalbnf(l, 1 - k - s));
}
// scale that puts a total like v at 2^40
__device__ __forceinline__ int res_scale(float v) {
  const int e = int((__float_as_uint(v) >> 23) & 255u);
  return e == 0 || e == 255 ? 40 : 40 - (e - 127);
}
__device__ __forceinline__ int res_scale(float2 v) { return res_scale(v.x); }
__device__ __forceinline__ int res_scale(double v) {
  const int e = int((static_cast<unsigned long long>(__double_as_longlong(v)) >> 52) & 2047ull);
  return e < 123 || e > 1923 ? 40 : 40 - (e - 1023);
}
