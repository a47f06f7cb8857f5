// tg_trig.cuh -- sine and cosine of FP64 angles on the integer pipes.
//
// An FP64 sincos is about 90 operations of a pipe that retires two per SM and
// clock; it bounded the gauge update (130 us at 1024^2 for 20 us of memory traffic) and took
// a sixth of a batch trajectory.  Here the angle is reduced by a 64 x 128 bit
// product with 2/pi and the Taylor series of sin(r)/r and cos(r), |r| <= pi/4, are
// summed by Horner's rule in 64-bit fixed point (32-bit where a coefficient is
// below 2^-32): about 170 integer instructions per angle.
// Series: sum (-z)^n / (2n+1)!, n <= 9, and sum (-z)^n / (2n)!, n <= 10, z = r^2 <=
// 0.617; the first terms left out are below 2^-72.  A product drops its low*low
// limbs and is at most 2 units of 2^-64 low; each factor z shrinks what came before,
// so the results are within 8 * 2^-64 absolute.  Relative accuracy (2 ulp) too:
//   * where no multiple of pi/2 was taken out, sin is formed as a * (sin(r)/r) in FP64;
//   * near the other multiples a part of a link below 2^-8 is left to the library, and
//     one of a Gaussian's angle, which is exact there, is formed as r * (sin(r)/r).
// |a| >= 2^20, Inf and NaN: fx_trig returns false.
#pragma once

#include "tg_fixed.cuh"

namespace tg {

typedef unsigned long long u64;

// floor(a b / 2^64), at most 2 low
TG_HD u64 mulhi_low(u64 a, u64 b) {
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
  return (u64)ah * bh + (((u64)ah * bl) >> 32) + (((u64)al * bh) >> 32);
}
TG_HD u64 mulhi_exact(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
TG_HD unsigned mulhi32(unsigned a, unsigned b) { return (unsigned)(((u64)a * b) >> 32); }

// u * 2^(-shift) as FP64
TG_HD double u64_scaled(u64 u, int shift) {
  const double d = (double)u;
  const int h = dbl_hi(d);
  return dbl_of(((u64)(unsigned)(h == 0 ? 0 : h - (shift << 20)) << 32) | dbl_lo(d));
}

struct FxTrig {
  u64 sn, cs;          // |sin a|, |cos a| * 2^64, at most 2^64 - 1
  bool neg_sn, neg_cs;  // their signs
  u64 ratio, vers;     // sin(r) / r and 1 - cos(r), * 2^64, of the reduced angle r
  bool reduced;        // a multiple of pi/2 was taken out (else |a| = r)
};

// From the reduced angle r >= 0 (u = r 2^64), its sign and the quadrant.
TG_HD FxTrig fx_trig_reduced(u64 u, bool neg_r, unsigned k, bool reduced) {
  const u64 z = mulhi_exact(u, u);
  const unsigned zh = (unsigned)(z >> 32);
  // sin(r) / r
  unsigned h = 0xca96u - mulhi32(zh, 0x98u);
  h = 0xd73f9fu - mulhi32(zh, h);
  h = 0xb092309du - mulhi32(zh, h);
  u64 p = 0x6b99159fd5ull - mulhi_low(z, h);
  p = 0x2e3bc74aad8eull - mulhi_low(z, p);
  p = 0xd00d00d00d00dull - mulhi_low(z, p);
  p = 0x222222222222222ull - mulhi_low(z, p);
  p = 0x2aaaaaaaaaaaaaabull - mulhi_low(z, p);
  // cos(r)
  unsigned w = 0xb41u - mulhi32(zh, 0x8u);
  w = 0xd73fau - mulhi32(zh, w);
  w = 0xc9cba54u - mulhi32(zh, w);
  u64 q = 0x8f76c77fcull - mulhi_low(z, w);
  q = 0x49f93edde28ull - mulhi_low(z, q);
  q = 0x1a01a01a01a02ull - mulhi_low(z, q);
  q = 0x5b05b05b05b05bull - mulhi_low(z, q);
  q = 0xaaaaaaaaaaaaaabull - mulhi_low(z, q);
  q = 0x8000000000000000ull - mulhi_low(z, q);
  FxTrig t;
  t.ratio = ~mulhi_low(z, p);
  t.vers = mulhi_low(z, q);
  const u64 s = mulhi_exact(u, t.ratio), c = ~t.vers;
  const bool odd = k & 1u;
  t.sn = odd ? c : s;
  t.cs = odd ? s : c;
  // quadrants 0 .. 3: sin = s, c, -s, -c; cos = c, -s, -c, s
  t.neg_sn = ((k & 2u) != 0) != (odd ? false : neg_r);
  t.neg_cs = (((k + 1u) & 2u) != 0) != (odd ? neg_r : false);
  t.reduced = reduced;
  return t;
}

TG_HD bool fx_trig(double a, FxTrig& out) {
  const int hi = dbl_hi(a);
  const int E = (int)(((unsigned)hi << 1) >> 21) - 1023;
  if (E >= 20) return false;
  const u64 m = ((u64)(((unsigned)hi & 0xfffffu) | 0x100000u) << 32) | dbl_lo(a);  // |a| = m 2^(E-52)
  // |a| 2/pi = m C 2^(E-180), C = 2/pi 2^128; the 128 bits above the lowest 64
  const u64 ch = 0xa2f9836e4e441529ull, cl = 0xfc2757d1f534ddc0ull;
  const u64 l1 = m * ch, h0 = mulhi_exact(m, cl);
  const u64 p1 = l1 + h0, p2 = mulhi_exact(m, ch) + (p1 < l1 ? 1ull : 0ull);
  const int sh = imin(52 - E, 63);  // 33 ... 63; below 2^-11 no bit reaches the quadrant or the rounding
  const u64 frac = (p1 >> sh) | (p2 << (64 - sh));
  const unsigned k = (unsigned)(p2 >> sh) + (unsigned)(frac >> 63);
  const bool neg = (long long)frac < 0;
  u64 f = neg ? 0 - frac : frac;
  f -= f >> 63;  // exactly 1/2: 2^-64 less, so that twice it fits
  const u64 ur = mulhi_exact(f << 1, 0xc90fdaa22168c234ull);  // times pi/2 2^63
  // no multiple taken out: r = |a| itself
  const u64 ua = (E >= -12) ? m << ((E + 12) & 63) : m >> imin(-(E + 12), 63);
  const bool reduced = k != 0;
  out = fx_trig_reduced(reduced ? ur : ua, reduced && neg, k, reduced);
  out.neg_sn = out.neg_sn != (hi < 0);
  return true;
}

// Results below 2^(kTrigSmall - 64) have less than FP64's relative accuracy.
constexpr int kTrigSmall = 56;

// half * sgn * (cos a, sin a) in FP64 and as limbs: one link (sgn = -1, 0 or 1).
TG_HD void fx_link_of(double a, int sgn, double2& w, FxLink& q) {
  FxTrig t;
  if (sgn != 0 && fx_trig(a, t) && !(t.reduced && ((t.sn < t.cs ? t.sn : t.cs) >> kTrigSmall) == 0)) {
    const bool flip = sgn < 0;
    const double wc = u64_scaled(t.cs, 65);
    w.x = (t.neg_cs != flip) ? -wc : wc;
    if (t.reduced) {
      const double d = u64_scaled(t.sn, 65);
      w.y = (t.neg_sn != flip) ? -d : d;
    } else {
      const double d = a * u64_scaled(t.ratio, 65);
      w.y = flip ? -d : d;
    }
    // u 2^-64 / 2 at the scale 2^60, to even: u / 32
    long long c = 2 * (long long)((t.cs >> 6) + ((t.cs >> 5) & 1)), s = 2 * (long long)((t.sn >> 6) + ((t.sn >> 5) & 1));
    if (t.neg_cs != flip) c = -c;
    if (t.neg_sn != flip) s = -s;
    const FxLimbs lc = fx_limbs(c), ls = fx_limbs(s);
    q.x = lc.hi;
    q.y = lc.lo;
    q.z = ls.hi;
    q.w = ls.lo;
    return;
  }
  double sn = 0, cs = 0;
#ifdef __CUDA_ARCH__
  sincos(a, &sn, &cs);
#else
  sn = sin(a);
  cs = cos(a);
#endif
  const double f = 0.5 * (double)sgn;
  w.x = f * cs;
  w.y = f * sn;
  q = (sgn == 0 && w.x == 0 && w.y == 0) ? fx_open_link() : to_fx_link(w);
}

// 1 - cos a
TG_HD double one_minus_cos(double a) {
  FxTrig t;
  if (!fx_trig(a, t)) return 1. - cos(a);
  if (!t.reduced) return u64_scaled(t.vers, 64);
  return t.neg_cs ? 1.0 + u64_scaled(t.cs, 64) : u64_scaled(0 - t.cs, 64);
}

// cos and sin of 2 pi (v + 1/2) 2^-53, v < 2^53
TG_HD void fx_sincos_turn(u64 v, double& cs, double& sn) {
  const u64 turn = (v << 11) + (1ull << 10), frac = turn << 2;
  const bool neg = (long long)frac < 0;
  const u64 f = neg ? 0 - frac : frac;  // frac is odd times 2^12: never exactly 1/2
  const unsigned k = (unsigned)(turn >> 62) + (unsigned)(frac >> 63);
  const FxTrig t = fx_trig_reduced(mulhi_exact(f << 1, 0xc90fdaa22168c234ull), neg, k, true);
  cs = u64_scaled(t.cs, 64);
  sn = u64_scaled(t.sn, 64);
  if ((f >> kTrigSmall) == 0) {  // f has 44 bits
    const double s = u64_scaled(f, 64) * 1.5707963267948966 * u64_scaled(t.ratio, 64);
    if (k & 1u) cs = s;
    else sn = s;
  }
  if (t.neg_cs) cs = -cs;
  if (t.neg_sn) sn = -sn;
}

}  // namespace tg
