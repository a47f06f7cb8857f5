// tg_device.cuh -- device functions shared by the single-lattice kernels
// (tg_kernels.cu) and the batched-chain kernel (tg_batch.cu): link
// coefficients, the staggered operator at one site, the force at one site, and
// the Philox generator.  One implementation, so both paths compute the same
// numbers for the same inputs.
#pragma once

#include <math.h>

#include "tg_launch.h"
#include "tg_trig.cuh"

namespace tg {

// ---------------------------------------------------------------------------
// Link coefficients  W_mu(s) = 0.5 * eta_mu(s) * bc_mu(s) * (cos A, sin A)
// eta_t(x) = (-1)^x, eta_x = 1 (hmc.c:914-921); bc_mu applies on the link that
// leaves the last slice (hmc.c:143-148, 165-170).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void write_links(const Geo& g, int bc_t, int bc_x, int s, double2 a, const LinkOut& o) {
  int t, x;
  site_tx(g, s, t, x);
  const int ft = ((x & 1) ? -1 : 1) * ((t == g.nt - 1) ? bc_t : 1), fx = (x == g.nx - 1) ? bc_x : 1;
  double2 w;
  FxLink q;
  fx_link_of(a.x, ft, w, q);
  if (o.Wt != nullptr) o.Wt[s] = w;
  o.Wt32[s] = make_float2((float)w.x, (float)w.y);
  o.Wtq[s] = q;
  fx_link_of(a.y, fx, w, q);
  if (o.Wx != nullptr) o.Wx[s] = w;
  o.Wx32[s] = make_float2((float)w.x, (float)w.y);
  o.Wxq[s] = q;
}

// ---------------------------------------------------------------------------
// The staggered operator at one site: hmc.c:132-183 for M (DAG = 0) and the
// true adjoint M^dagger = m - D(-mu) (DAG = 1).  MU0 drops the e^{+-mu}
// factors (mu = 0): 18 FMA/MUL per site instead of 22.  This is the FP32
// operator, and the FP64 one where fx_dslash (tg_fixed.cuh) is out of range.
// ---------------------------------------------------------------------------
template <typename R, int DAG, bool MU0>
__device__ __forceinline__ C2<R> dslash_vals(const OpK<R>& k, C2<R> pc, C2<R> ptu, C2<R> ptd, C2<R> pxu, C2<R> pxd,
                                             C2<R> wt, C2<R> wtd, C2<R> wx, C2<R> wxd) {
  // pc = in(s); ptu/ptd = in(s+t)/in(s-t); pxu/pxd = in(s+x)/in(s-x);
  // wt = Wt(s), wtd = Wt(s-t), wx = Wx(s), wxd = Wx(s-x)
  C2<R> o = mk<R>(k.m * pc.x, k.m * pc.y);
  if (MU0) {
    if (DAG == 0) {
      cmac<R>(o, wt, ptu);
      cmsc<R>(o, wtd, ptd);
    } else {
      cnmac<R>(o, wt, ptu);
      cjmac<R>(o, wtd, ptd);
    }
  } else {
    C2<R> ft = cmul<R>(wt, ptu);
    C2<R> bt = cjmul<R>(wtd, ptd);
    o.x = fma(k.cf, ft.x, o.x);
    o.y = fma(k.cf, ft.y, o.y);
    o.x = fma(k.cb, bt.x, o.x);
    o.y = fma(k.cb, bt.y, o.y);
  }
  if (DAG == 0) {
    cmac<R>(o, wx, pxu);
    cmsc<R>(o, wxd, pxd);
  } else {
    cnmac<R>(o, wx, pxu);
    cjmac<R>(o, wxd, pxd);
  }
  return o;
}

// The links an operator of precision R reads: FP32 values, or the limbs of the
// FP64 operator.
template <typename R> struct LkT;
template <> struct LkT<float> { using type = float2; };
template <> struct LkT<double> { using type = FxLink; };
template <typename R> using Lk = typename LkT<R>::type;

// The FP64 form of a site that fx_dslash refuses.  Most such sites have zeros for
// operands (a vector that is zero in places, as point sources are): they give zero
// without the FP64 pipe, which doubled the time of a zero vector's apply.
template <int DAG, bool MU0>
__device__ __forceinline__ double2 dslash_wide(const OpK<double>& k, double2 pc, double2 ptu, double2 ptd, double2 pxu,
                                               double2 pxd, FxLink wt, FxLink wtd, FxLink wx, FxLink wxd) {
  const bool zero = pc.x == 0 && pc.y == 0 && ptu.x == 0 && ptu.y == 0 && ptd.x == 0 && ptd.y == 0 && pxu.x == 0 &&
                    pxu.y == 0 && pxd.x == 0 && pxd.y == 0;
  // (a constant or a link that is not finite makes it NaN)
  if (zero && fx_finite(k, wt, wtd, wx, wxd)) return make_double2(0.0, 0.0);
  return dslash_vals<double, DAG, MU0>(k, pc, ptu, ptd, pxu, pxd, fx_link_value(wt), fx_link_value(wtd),
                                       fx_link_value(wx), fx_link_value(wxd));
}

// The operator at site s = (t, x) with operands from ld; own = the operand at s.
template <typename R, int DAG, bool MU0, class Ld>
__device__ __forceinline__ C2<R> dslash_ld(const Geo& g, const OpK<R>& k, Ld& ld, const Lk<R>* __restrict__ Wt,
                                           const Lk<R>* __restrict__ Wx, int s, int t, int x, C2<R>& own) {
  const Nbr n = neighbours(g, s, t, x);
  own = ld(s);
  const C2<R> tu = ld(n.tp), td = ld(n.tm), xu = ld(n.xp), xd = ld(n.xm);
  const Lk<R> wt = Wt[s], wtd = Wt[n.tm], wx = Wx[s], wxd = Wx[n.xm];
  if constexpr (sizeof(R) == 4) {
    return dslash_vals<R, DAG, MU0>(k, own, tu, td, xu, xd, wt, wtd, wx, wxd);
  } else {
    double2 o;
    if (!fx_dslash<DAG, MU0>(k, to_fx(own), to_fx(tu), to_fx(td), to_fx(xu), to_fx(xd), wt, wtd, wx, wxd, o))
      o = dslash_wide<DAG, MU0>(k, own, tu, td, xu, xd, wt, wtd, wx, wxd);
    return o;
  }
}

template <typename R, int DAG, bool MU0>
__device__ __forceinline__ C2<R> dslash_at(const Geo& g, const OpK<R>& k, const C2<R>* __restrict__ in,
                                           const Lk<R>* __restrict__ Wt, const Lk<R>* __restrict__ Wx, int s) {
  int t, x;
  site_tx(g, s, t, x);
  auto ld = [&](int i) { return in[i]; };
  C2<R> own;
  return dslash_ld<R, DAG, MU0>(g, k, ld, Wt, Wx, s, t, x, own);
}

template <typename R> __device__ __forceinline__ C2<R> shfl_down1(C2<R> v) {
  return mk<R>(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}
template <typename R> __device__ __forceinline__ C2<R> shfl_up1(C2<R> v) {
  return mk<R>(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}

// Force pieces at one site (momentum_step, hmc.c:504-661):
//   gauge   (Nf/g) sin A                                           (507-510)
//   pf      2 Im W (e^{mu} conj(Mchi(s)) chi(s+mu) - e^{-mu} conj(chi(s)) Mchi(s+mu))   (517-576)
//   noise   -(e^{mu} - e^{-mu}) Im W conj(n(s)) n(s+t), t links only  (608-661)
struct ForcePieces {
  double2 g, pf, md;
};

// The gauge force's sin A comes from the link coefficient the same gauge step
// wrote: W = f e^{iA} with f = +-1/2, so sin A = Im W / f exactly (f and 1/f
// are powers of two).  A link with f = 0 (open boundary) takes sin A itself.
__device__ __forceinline__ ForcePieces force_site(const Geo& g, int bc_t, int bc_x, double ep, double em,
                                                  const double2* A, const double2* Wt, const double2* Wx,
                                                  const double2* chi, const double2* Mchi, const double2* noise,
                                                  int s) {
  int t, x;
  site_tx(g, s, t, x);
  Nbr n = neighbours(g, s, t, x);
  ForcePieces f;
  const double bt = (t == g.nt - 1) ? (double)bc_t : 1.0;
  const double bx = (x == g.nx - 1) ? (double)bc_x : 1.0;
  const double inv_ft = ((x & 1) ? -2.0 : 2.0) * bt, inv_fx = 2.0 * bx;
  f.g.x = (bt != 0.0) ? Wt[s].y * inv_ft : sin(A[s].x);
  f.g.y = (bx != 0.0) ? Wx[s].y * inv_fx : sin(A[s].y);
  f.pf = make_double2(0, 0);
  f.md = make_double2(0, 0);
  if (chi != nullptr) {
    double2 c0 = chi[s], m0 = Mchi[s];
    double2 ct = chi[n.tp], mt = Mchi[n.tp];
    double2 cx = chi[n.xp], mx = Mchi[n.xp];
    // e1*conj(m0)*c_next - e2*conj(c0)*m_next
    double2 q1 = cjmul<double>(m0, ct), q2 = cjmul<double>(c0, mt);
    double2 qt = make_double2(ep * q1.x - em * q2.x, ep * q1.y - em * q2.y);
    double2 r1 = cjmul<double>(m0, cx), r2 = cjmul<double>(c0, mx);
    double2 qx = make_double2(r1.x - r2.x, r1.y - r2.y);
    double2 wt = Wt[s], wx = Wx[s];
    f.pf.x = 2.0 * fma(wt.x, qt.y, wt.y * qt.x);
    f.pf.y = 2.0 * fma(wx.x, qx.y, wx.y * qx.x);
  }
  if (noise != nullptr) {
    double d = ep - em;
    double2 q = cjmul<double>(noise[s], noise[n.tp]);
    double2 wt = Wt[s];
    f.md.x = -d * fma(wt.x, q.y, wt.y * q.x);
  }
  return f;
}

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11), counter = (site,
// stream, trajectory lo, trajectory hi), key = seed.  Each draw gives two
// 53-bit uniforms in (0,1) -> one Box-Muller pair.
__device__ __forceinline__ uint4 philox4x32(uint4 c, uint2 k) {
#pragma unroll
  for (int i = 0; i < 10; i++) {
    unsigned hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    unsigned hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}

__device__ __forceinline__ double u53(unsigned hi, unsigned lo) {
  // ((hi:lo) >> 11 + 0.5) * 2^-53, strictly inside (0,1)
  unsigned long long v = ((unsigned long long)hi << 21) ^ (lo >> 11);
  return ((double)v + 0.5) * 1.1102230246251565e-16;
}

__device__ __forceinline__ double2 philox_gauss_pair(unsigned long long seed, unsigned long long tr, unsigned site,
                                                     unsigned stream_id) {
  uint4 r = philox4x32(make_uint4(site, stream_id, (unsigned)tr, (unsigned)(tr >> 32)),
                       make_uint2((unsigned)seed, (unsigned)(seed >> 32)));
  double u1 = u53(r.x, r.y);
  double rad = sqrt(-2.0 * log(u1));
  double sn, cs;
  fx_sincos_turn(((unsigned long long)r.z << 21) ^ (r.w >> 11), cs, sn);  // 2 pi u53(r.z, r.w)
  return make_double2(rad * cs, rad * sn);
}

__device__ __forceinline__ double philox_uniform1(unsigned long long seed, unsigned long long tr, unsigned stream_id) {
  uint4 r = philox4x32(make_uint4(0xffffffffu, stream_id, (unsigned)tr, (unsigned)(tr >> 32)),
                       make_uint2((unsigned)seed, (unsigned)(seed >> 32)));
  return u53(r.x, r.y);
}

}  // namespace tg
