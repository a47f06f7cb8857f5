// tg_scalar.cuh -- the scalar steps between two passes of a CG iteration, with
// short dependent chains.  On GB300 an FP64 add has a latency of 55 clocks, a
// shuffle-and-add tree step 86 (150 with eight warps on an SM, whose FP64 pipe
// retires two operations per clock), an FP64 division 574; an integer warp
// reduction (REDUX) 30-50 and a 64-bit integer add 15 (measured).  So
//   * sums of squares are added as 64-bit integers at a scale that follows the
//     last total of their kind (FxTotal): exact within the sum, independent of
//     its order, resolution 2^-60 of that total;
//   * the quotient of two sums is formed from a reciprocal that is computed
//     beforehand, or by Newton's iteration, with one residual correction.
// The conversions and the quotient are host-callable for the tests.
#pragma once

#include "tg_fixed.cuh"

namespace tg {

// a / b for b > 0 normal, given inv = 1 / b to 45 bits or better: q = a inv,
// corrected once by the residual a - b q.
TG_HD double div_corrected(double a, double b, double inv) {
  const double q = a * inv;
  return fma(fma(-b, q, a), inv, q);
}

// a / b, b > 0, given inv = 1 / b rounded: the same, where inv has not overflowed or
// come near it (b < 2^-1000: plain division).
TG_HD double div_prepared(double a, double b, double inv) {
  return inv < 1.0715086071862673e301 ? div_corrected(a, b, inv) : a / b;  // 2^1000
}

// a / b by Newton's iteration on the reciprocal (x' = x + x (1 - b x), which
// doubles the correct bits) from an FP32 reciprocal of b's mantissa, then the
// residual correction (without CORRECT, for a quotient that is rounded to FP32,
// a / b to 2^-44).  b outside [2^-900, 2^900], zero, Inf or NaN: plain
// division.
template <bool CORRECT = true> TG_HD double div_newton(double a, double b) {
  const int hb = dbl_hi(b);
  const int e = hb >> 20;  // sign and exponent field: 123 ... 1923 for the accepted b
  if (e < 123 || e > 1923) return a / b;
  union { unsigned u; float f; } m, r;
  m.u = 0x3f800000u | (((unsigned)hb & 0xfffffu) << 3) | (dbl_lo(b) >> 29);  // in [1, 2)
  r.f = 1.0f / m.f;                                                         // in [1/2, 1]
  // the same value as FP64, times 2^(1023 - e)
  const unsigned long long x =
      ((unsigned long long)((r.u >> 3) + ((1023u - 127u) << 20) + ((1023u - (unsigned)e) << 20)) << 32) |
      (unsigned)(r.u << 29);
  double inv = dbl_of(x);
  inv = fma(inv, fma(-b, inv, 1.0), inv);
  return CORRECT ? div_corrected(a, b, inv) : a * inv;
}

// ---------------------------------------------------------------------------
// Sums of non-negative terms as integers.  ref: exponent field of the last total of
// the kind (0: none); a term t is added as rint(t * 2^(61 - (ref - 1023))), so
// the total comes out near 2^61 and a term's rounding is 2^-62 of it.  Terms are
// added by limbs of 26, 26 and 11 bits; one of 2^63 or more (or not finite)
// gives a top limb of 2^17.  A total below 2^58 or with a top limb of 2^17 - 64
// or more is refused: the sum is then taken again in FP64.
// ---------------------------------------------------------------------------
constexpr unsigned kFxTopRefused = 1u << 17;
constexpr int kFxRefMin = 200, kFxRefMax = 1900;

struct FxTerm {
  unsigned low, mid, top;
};
TG_HD FxTerm fx_split(unsigned long long q, bool refused) {
  return FxTerm{(unsigned)q & 0x3ffffffu, (unsigned)(q >> 26) & 0x3ffffffu,
                refused ? kFxTopRefused : (unsigned)(q >> 52)};
}
TG_HD int fx_total_ref(double total) {
  const int e = (int)((unsigned)dbl_hi(total) >> 20);  // a negative total or NaN is out of range too
  return (e >= kFxRefMin && e <= kFxRefMax) ? e : 0;
}
TG_HD unsigned long long fx_shift(unsigned long long m, int sh) {
  if (sh >= 0) return m << (sh & 63);
  return ((m >> (imin(-sh, 63) - 1)) + 1) >> 1;  // to nearest
}
// an FP64 term; v >= 0 or NaN
TG_HD FxTerm fx_term(double v, int ref) {
  const int sh = ((dbl_hi(v) >> 20) & 0x7ff) - ref + 9;
  const unsigned long long m = (((unsigned long long)((unsigned)dbl_hi(v) & 0xfffffu) | 0x100000ull) << 32) | dbl_lo(v);
  // zero and denormal terms (exponent field 0) shift out: ref >= 200
  return fx_split(fx_shift(m, sh), ref == 0 || sh > 10);
}
// an FP32 term; v >= 0 or NaN
TG_HD FxTerm fx_term(float v, int ref) {
  union { float f; unsigned u; } b;
  b.f = v;
  const int e = (int)((b.u >> 23) & 0xffu);
  // a denormal has exponent 1 and no leading one (a sum of r^2 in FP32 may lie below 2^-126)
  const int sh = (e == 0 ? 1 : e) + 934 - ref;
  const unsigned long long m = (unsigned long long)((b.u & 0x7fffffu) | (e == 0 ? 0u : 0x800000u));
  return fx_split(fx_shift(m, sh), ref == 0 || e == 255 || (sh > 39 && (m >> (sh < 63 ? 63 - sh : 0)) != 0));
}
// The total as FP64 from its three limbs: low + mid 2^26 + top 2^52 (low, mid < 2^32).
TG_HD bool fx_total_value(unsigned low, unsigned mid, unsigned top, int ref, double& total) {
  const unsigned long long q = ((unsigned long long)top << 46) + ((low + ((unsigned long long)mid << 26)) >> 6);
  const double d = (double)(long long)q;
  total = dbl_of(((unsigned long long)(unsigned)(dbl_hi(d) + (ref - 1078) * 1048576) << 32) | dbl_lo(d));
  return q >= (1ull << 52) && top < kFxTopRefused - 64 && ref != 0;
}

// The bits of a double that is not negative (a norm, a stopping threshold), which
// compare as it does, NaN above all: a NaN may have its sign set (an invalid operation's has).
TG_HD long long norm_bits(double v) {
  return (long long)(((unsigned long long)((unsigned)dbl_hi(v) & 0x7fffffffu) << 32) | dbl_lo(v));
}

// The verdict on |r|^2 = rn after a CG iteration: a status, or -1 to go on
// (hmc.c:381-386).
TG_HD int cg_verdict(double rn, double stop, double limit, bool last) {
  const long long b = norm_bits(rn);
  if (b > norm_bits(INFINITY)) return TG_E_NAN;
  if (b < norm_bits(stop)) return TG_OK;
  if (b > norm_bits(limit)) return TG_E_DIVERGED;
  return last ? TG_E_NOCONV : -1;
}
// The mixed solvers' test for a reliable update, besides the count of iterations
TG_HD bool cg_update_due(double rn, double stop, double drop, double limit) {
  const long long b = norm_bits(rn);
  return b < norm_bits(stop) || b < norm_bits(drop) || b > norm_bits(limit);
}

#ifdef __CUDACC__
// A warp's partial: low + mid 2^26 in x, the top limbs in y.
__device__ __forceinline__ longlong2 fx_warp_partial(FxTerm t) {
  const unsigned slo = __reduce_add_sync(0xffffffffu, t.low), smid = __reduce_add_sync(0xffffffffu, t.mid),
                 stop = __reduce_add_sync(0xffffffffu, t.top);
  return make_longlong2((long long)(slo + ((unsigned long long)smid << 26)), (long long)stop);
}
// The total of n warps' partials (n <= 512), by one warp; the same in every lane.
__device__ __forceinline__ bool fx_partials_total(const longlong2* part, int n, int ref, double& total) {
  const int lane = threadIdx.x & 31;
  longlong2 v = make_longlong2(0, 0);
  if (lane < n) v = part[lane];
  for (int j = lane + 32; j < n; j += 32) {
    const longlong2 w = part[j];
    v.x += w.x;
    v.y += w.y;
  }
  const unsigned slo = __reduce_add_sync(0xffffffffu, (unsigned)v.x & 0x3ffffffu),
                 smid = __reduce_add_sync(0xffffffffu, (unsigned)(v.x >> 26) & 0x3ffffffu),
                 stop = __reduce_add_sync(0xffffffffu, (unsigned)(v.x >> 52) + (unsigned)v.y);
  return fx_total_value(slo, smid, stop, ref, total);
}
#endif

}  // namespace tg
