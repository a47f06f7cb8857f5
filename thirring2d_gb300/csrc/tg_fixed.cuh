// tg_fixed.cuh -- the FP64 staggered operator on the integer pipes.
//
// GB300 retires about two FP64 operations per SM and clock and 64 32x32+64-bit
// integer multiply-adds (measured: DFMA 1.7, IMAD.WIDE 55-64 lanes per SM and
// clock), so the 16 real products of one operator site cost 10 clocks as DFMA
// and under one as integer limb products.  A site is therefore computed in
// block floating point, with FP64 in and out:
//   * a complex operand is two 60-bit two's-complement integers at the larger
//     exponent of its two parts (to_fx);
//   * a link, |W| <= 1/2, is two 60-bit integers at the scale 2^60, converted
//     once per gauge update (to_fx_link) into signed 32-bit limbs
//     (high, low), 16 bytes as the double2 it replaces;
//   * the five operands of a site are shifted to their largest exponent, the
//     products taken limb by limb (high*high and the two cross products; the
//     dropped low*low is under 1/4 unit) and added exactly in 64 bits, and the
//     sum is rounded once to FP64.
// With P the largest |part| among the five operands (times its operator
// constant), the integer sum is within 4 units of 2^-56 P of the exact value;
// FP64's own order of nine roundings is within about 9 * 2^-54 P.  The
// alignment is per site, so a small operand beside larger ones loses no more
// than it does to FP64 addition, and the result is a function of the site's
// operands alone: every path that computes a site returns the same bits.
// This is a bound for the site, not for each component: a part of a result far
// below P (the imaginary part for a real vector on a field next to the cold one; a part of
// an operand 2^53 times below its other) has P's absolute accuracy, where multiply-adds in
// FP64 would keep more of it.  (Links with a part below 2^-21 in the FP64 form instead: a
// 1024^2 field of Gaussian angles of 0.3 has five, and they cost its trajectory 10%.)
//
// Measured on GB300: the FP64 apply at 1024^2 32 -> 19.2 us (0.3 of it the test for open
// boundaries) and at 2048^2 135 -> 79 us, the FP64 CG iteration at 1024^2 86.8 -> 58.7 us (52.8 with the
// rows prefetched, tg_stencil.cuh); error against exact arithmetic 1.1e-16 relative (FP64 FMA order: 1.4e-16).
//
// Exponents outside [kFxEmin, kFxEmax] (operands all zero, denormal, huge, Inf
// or NaN), operator constants that are not finite, and links that are not
// finite (marked by bit 0 of the real low limb) take the FP64 form: fx_dslash
// returns false and the caller computes the site in FP64.
#pragma once

#include <math.h>
#include <string.h>

#include "tg_internal.cuh"

namespace tg {

constexpr int kFxEmin = 200, kFxEmax = 2020;

#define TG_HD __host__ __device__ __forceinline__

TG_HD int dbl_hi(double v) {
#ifdef __CUDA_ARCH__
  return __double2hiint(v);
#else
  long long b;
  memcpy(&b, &v, 8);
  return (int)(b >> 32);
#endif
}
TG_HD unsigned dbl_lo(double v) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(v);
#else
  long long b;
  memcpy(&b, &v, 8);
  return (unsigned)b;
#endif
}
TG_HD double dbl_of(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double v;
  memcpy(&v, &b, 8);
  return v;
#endif
}
TG_HD int clz64(unsigned long long a) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}

// One link: signed limbs (real high, real low, imaginary high, imaginary low).
using FxLink = int4;

// A complex operand: value (re + i im) * 2^(e - 1082), |re|, |im| < 2^60.
struct FxC {
  long long re, im;
  int e;
};

// a * 2^32 limb split with a signed low limb: v = hi * 2^32 + lo
struct FxLimbs {
  int hi, lo;
};
TG_HD FxLimbs fx_limbs(long long v) {
  FxLimbs l;
  l.lo = (int)v;
  l.hi = (int)(v >> 32) + (int)((unsigned)v >> 31);
  return l;
}

TG_HD int imin(int a, int b) { return a < b ? a : b; }
TG_HD int imax(int a, int b) { return a > b ? a : b; }

// 60-bit magnitude of a double at exponent e >= its own, in one's complement
// for negative values (off by at most 2^-60 of 2^(e - 1022)).  Zero and
// denormal parts (exponent field 0) carry a stray hidden bit here; it is
// shifted out, because the site's exponent is at least kFxEmin > 64.
TG_HD long long fx_part(double v, int ev, int e) {
  const int h = dbl_hi(v);
  unsigned long long m = ((unsigned long long)(((unsigned)h & 0xfffffu) | 0x100000u) << 32) | dbl_lo(v);
  m = (m << 7) >> imin(e - ev, 63);
  return (long long)(m ^ (unsigned long long)(long long)(h >> 31));
}

TG_HD FxC to_fx(double2 v) {
  FxC f;
  const int er = (int)(((unsigned)dbl_hi(v.x) << 1) >> 21), ei = (int)(((unsigned)dbl_hi(v.y) << 1) >> 21);
  f.e = imax(er, ei);
  f.re = fx_part(v.x, er, f.e);
  f.im = fx_part(v.y, ei, f.e);
  return f;
}

// The operand as FP64 again, for the FP64 form where only the block-floating
// one was kept: operands that are not finite give NaN, zero and denormal ones 0.
TG_HD double2 fx_value(const FxC& f) {
  double2 v;
  if (f.e == 0) {
    v.x = v.y = 0.0;
  } else if (f.e == 2047) {
    v.x = v.y = dbl_of(0x7ff8000000000000ull);
  } else {
    v.x = ldexp((double)f.re, f.e - 1082);
    v.y = ldexp((double)f.im, f.e - 1082);
  }
  return v;
}

// W (|parts| <= 1/2) at the scale 2^60, rounded to even multiples; a part that
// is not finite sets bit 0 of the real low limb.
TG_HD FxLink to_fx_link(double2 w) {
  const bool bad = !(fabs(w.x) <= 1.0) || !(fabs(w.y) <= 1.0);
  const double s = 576460752303423488.0;  // 2^59
  const FxLimbs r = fx_limbs(bad ? 0 : 2 * (long long)rint(w.x * s)), i = fx_limbs(bad ? 0 : 2 * (long long)rint(w.y * s));
  FxLink l;
  l.x = r.hi;
  l.y = bad ? 1 : r.lo;
  l.z = i.hi;
  l.w = i.lo;
  return l;
}
// A link across an open boundary, W = 0, is marked too, and says so in bit 0 of the
// imaginary low limb: the operand behind it does not contribute and must not set the scale
// of the site's sum (beside one 2^60 times the others nothing would be left of them).
TG_HD FxLink fx_open_link() {
  FxLink l;
  l.x = l.z = 0;
  l.y = l.w = 1;
  return l;
}
// ... and back, for the FP64 form
TG_HD double2 fx_link_value(FxLink l) {
  const double s = 1.0 / 1152921504606846976.0;  // 2^-60
  double2 w;
  w.x = (double)((long long)l.x * 4294967296LL + l.y) * s;
  w.y = (double)((long long)l.z * 4294967296LL + l.w) * s;
  if (l.y & 1) w.x = w.y = (l.w & 1) ? 0.0 : dbl_of(0x7ff8000000000000ull);
  return w;
}

// Marked and not finite (bit 0)
TG_HD int fx_link_bad(FxLink l) { return l.y & ~l.w; }

// Operator constants.  out = m in + cf Wt in(+t) + cb conj(Wt(-t)) in(-t) + ...;
// besides the FP64 values, m as 60-bit limbs at the scale 2^60 with its
// exponent me, and |cf|, |cb| as 62-bit limbs (values in [1/2, 1)) with theirs.
// emin: kFxEmin, or above every exponent when a constant is not finite.
template <> struct OpK<double> {
  double m, cf, cb;
  int mu0;
  FxLimbs fm, ff, fb;
  int me, fe, be, emin;
};

TG_HD OpK<double> make_opk(double m, double cf, double cb, bool mu0) {
  OpK<double> k;
  k.m = m;
  k.cf = cf;
  k.cb = cb;
  k.mu0 = mu0;
  // frexp by hand (the same on host and device): exponent field of a normal number
  auto split = [](double v, int bits, FxLimbs& l, int& ex) {
    const int e = (int)(((unsigned)dbl_hi(v) << 1) >> 21);
    if (e == 0) {  // 0 or denormal: as 0
      l.hi = l.lo = 0;
      ex = -4096;
      return;
    }
    const unsigned long long mant =
        (((unsigned long long)((unsigned)dbl_hi(v) & 0xfffffu) | 0x100000ull) << 32) | dbl_lo(v);  // 53 bits
    long long q = (long long)(mant << (bits - 53));
    if (dbl_hi(v) < 0) q = -q;
    l = fx_limbs(q);
    ex = e - 1022;  // v = (mant * 2^-53) * 2^ex, mant * 2^-53 in [1/2, 1)
  };
  split(m, 60, k.fm, k.me);
  split(fabs(cf), 62, k.ff, k.fe);
  split(fabs(cb), 62, k.fb, k.be);
  const bool ok = fabs(m) <= 1e300 && fabs(cf) <= 1e300 && fabs(cb) <= 1e300 && fabs(cf) >= 1e-300 &&
                  fabs(cb) >= 1e-300 && (m == 0.0 || fabs(m) >= 1e-300);
  k.emin = ok ? kFxEmin : (1 << 24);
  return k;
}

TG_HD long long mul_wide(int a, int b) { return (long long)a * (long long)b; }

// w * c for a 62-bit constant c in [1/2, 1): limbs at the scale 2^60 again
TG_HD FxLimbs fx_scale(int wh, int wl, FxLimbs c) {
  const long long x = mul_wide(wh, c.lo) + mul_wide(wl, c.hi) + 0x80000000LL;
  return fx_limbs((mul_wide(wh, c.hi) + (x >> 32)) * 4);
}
TG_HD FxLink fx_scale_link(FxLink w, FxLimbs c) {
  const FxLimbs r = fx_scale(w.x, w.y, c), i = fx_scale(w.z, w.w, c);
  FxLink o;
  o.x = r.hi;
  o.y = r.lo;
  o.z = i.hi;
  o.w = i.lo;
  return o;
}

// Sums of limb products, positive and negative terms apart (a product then
// needs no negation): high*high and the cross products.  Worst case 8 link
// products and the mass: under 2^63 in each.
struct FxAcc {
  long long ph, px, nh, nx;
};

template <bool NEG> TG_HD void fx_mac(FxAcc& a, int wh, int wl, FxLimbs v) {
  if (NEG) {
    a.nh += mul_wide(wh, v.hi);
    a.nx += mul_wide(wh, v.lo);
    a.nx += mul_wide(wl, v.hi);
  } else {
    a.ph += mul_wide(wh, v.hi);
    a.px += mul_wide(wh, v.lo);
    a.px += mul_wide(wl, v.hi);
  }
}

// (x, y) += (NEG ? -1 : 1) * (CONJ ? conj(w) : w) * (v >> d)
template <bool CONJ, bool NEG> TG_HD void fx_cmac(FxAcc& x, FxAcc& y, FxLink w, const FxC& v, int d) {
  d = imin(d, 63);
  const FxLimbs r = fx_limbs(v.re >> d), i = fx_limbs(v.im >> d);
  fx_mac<NEG>(x, w.x, w.y, r);
  fx_mac<CONJ == NEG>(x, w.z, w.w, i);
  fx_mac<NEG>(y, w.x, w.y, i);
  fx_mac<CONJ != NEG>(y, w.z, w.w, r);
}

// The sum as FP64 (round to nearest), in units of 2^(e - 1078).  The conversion
// runs on the FP64 pipe (2 per SM and clock), its 20 integer instructions would
// run on the ALUs, which bound the operator: apply at 2048^2 78.5 against 84.1 us.
TG_HD double fx_round(const FxAcc& a, int e) {
  const long long t = (a.ph - a.nh) + ((a.px - a.nx + 0x80000000LL) >> 32);
  const double d = (double)t;
  const int h = dbl_hi(d);
  return dbl_of(((unsigned long long)(unsigned)(h == 0 ? 0 : h + ((e - 1078) << 20)) << 32) | dbl_lo(d));
}

// The operator at one site (dslash_vals of tg_device.cuh) from block-floating
// operands; false: out of range, out is not set.
template <int DAG, bool MU0>
TG_HD bool fx_dslash(const OpK<double>& k, const FxC& pc, const FxC& ptu, const FxC& ptd, const FxC& pxu,
                     const FxC& pxd, FxLink wt, FxLink wtd, FxLink wx, FxLink wxd, double2& out) {
  const int ec = pc.e + k.me;
  int etu = MU0 ? ptu.e : ptu.e + k.fe, etd = MU0 ? ptd.e : ptd.e + k.be, exu = pxu.e, exd = pxd.e;
  int bad = (wt.y | wtd.y | wx.y | wxd.y) & 1;
  if (bad) {  // not finite, or operands behind open boundaries (of which one that is not finite makes the site NaN)
    bad = (fx_link_bad(wt) | fx_link_bad(wtd) | fx_link_bad(wx) | fx_link_bad(wxd)) & 1;
    if ((wt.w & wt.y & 1) && ptu.e <= kFxEmax) etu = -4096;
    if ((wtd.w & wtd.y & 1) && ptd.e <= kFxEmax) etd = -4096;
    if ((wx.w & wx.y & 1) && pxu.e <= kFxEmax) exu = -4096;
    if ((wxd.w & wxd.y & 1) && pxd.e <= kFxEmax) exd = -4096;
  }
  const int E = imax(imax(imax(etu, etd), imax(exu, exd)), ec);
  // the largest operand exponent itself: E can lie below it by a constant's
  const int eraw = MU0 ? imax(E, pc.e) : imax(imax(imax(etu - k.fe, etd - k.be), imax(exu, exd)), pc.e);
  const bool ok = E >= k.emin && E <= kFxEmax && eraw <= kFxEmax && !bad;
  FxAcc x = {0, 0, 0, 0}, y = {0, 0, 0, 0};
  {
    const int d = imin(E - ec, 63);
    fx_mac<false>(x, k.fm.hi, k.fm.lo, fx_limbs(pc.re >> d));
    fx_mac<false>(y, k.fm.hi, k.fm.lo, fx_limbs(pc.im >> d));
  }
  fx_cmac<false, DAG != 0>(x, y, MU0 ? wt : fx_scale_link(wt, k.ff), ptu, E - etu);
  fx_cmac<true, DAG == 0>(x, y, MU0 ? wtd : fx_scale_link(wtd, k.fb), ptd, E - etd);
  fx_cmac<false, DAG != 0>(x, y, wx, pxu, E - exu);
  fx_cmac<true, DAG == 0>(x, y, wxd, pxd, E - exd);
  out.x = fx_round(x, E);
  out.y = fx_round(y, E);
  return ok;
}

// For a site that fx_dslash refused: nothing makes the products of zeros NaN.
TG_HD bool fx_finite(const OpK<double>& k, FxLink wt, FxLink wtd, FxLink wx, FxLink wxd) {
  return k.emin == kFxEmin && !((fx_link_bad(wt) | fx_link_bad(wtd) | fx_link_bad(wx) | fx_link_bad(wxd)) & 1);
}
// Zero of either sign: exponent 0 and only the stray bit (a denormal has mantissa bits besides it).
TG_HD bool fx_zero(const FxC& f) {
  return f.e == 0 && (((f.re ^ (f.re >> 63)) | (f.im ^ (f.im >> 63))) ^ (1LL << 59)) == 0;
}

}  // namespace tg
