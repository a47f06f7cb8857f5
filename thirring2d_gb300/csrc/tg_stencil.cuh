// tg_stencil.cuh -- the warp column march of the staggered operator, shared
// by the launch-per-iteration kernels (tg_kernels.cu) and the persistent
// solver (tg_pcg.cu), in two forms:
//   march_segment         operands loaded into registers as the march needs them
//   march_segment_staged  rows of the next chunks staged in shared memory by
//                         TMA bulk copies (cp.async.bulk + mbarrier) while the
//                         current chunk computes
#pragma once

#include "tg_device.cuh"

namespace tg {

// A lane's place in strip xw: columns x0 .. x0 + last are the strip's, x the lane's (the
// lanes beyond repeat the last one), xle and xre the columns beside the strip.
struct Strip {
  int x0, last, x, xle, xre;
};
TG_HD Strip strip_of(int nx, int xw, int lane) {
  Strip p;
  p.x0 = xw << 5;
  p.last = imin(nx - p.x0, 32) - 1;
  p.x = p.x0 + imin(lane, p.last);
  p.xle = (p.x0 == 0) ? nx - 1 : p.x0 - 1;
  p.xre = (p.x0 + p.last + 1 == nx) ? 0 : p.x0 + p.last + 1;
  return p;
}

// One row t of a warp's FP32 march: the operator at the sites (t, x0 + lane), lane
// <= last, from psi(t-1) = pm, psi(t) = pc, psi(t+1) = pp and the links, with the
// operand across the warp's edge pe (used by lanes 0 and last) and the x link
// entering column x0 we (used by lane 0).  Rotates pm, pc, wtm for row t+1.
template <typename R, int DAG, bool MU0, class Epi>
__device__ __forceinline__ void march_row(const OpK<R>& k, int s, int lane, int last, C2<R>& pm, C2<R>& pc, C2<R>& wtm,
                                          C2<R> pp, C2<R> wt, C2<R> wx, C2<R> pe, C2<R> we, Epi& epi) {
  C2<R> pr = shfl_down1<R>(pc);
  C2<R> pl = shfl_up1<R>(pc);
  C2<R> wl = shfl_up1<R>(wx);
  if (lane == last) pr = pe;
  if (lane == 0) {
    pl = pe;
    wl = we;
  }
  const C2<R> o = dslash_vals<R, DAG, MU0>(k, pc, pp, pm, pr, pl, wt, wtm, wx, wl);
  if (lane <= last) epi(s, o, pc);
  pm = pc;
  pc = pp;
  wtm = wt;
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

template <typename R> __device__ __forceinline__ C2<R> shfl_c2(C2<R> v, int src) {
  return mk<R>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// The operands across the warp's two edges for rows t .. t+kMarchT-1, fetched
// once by the first lanes: lane i < kMarchT the operand left of x0 in row t+i
// (and, in ew, the x link entering x0), lane kMarchT+i the operand right of
// x0+31.  Shuffles later hand them to lanes 0 and 31, so no lane fetches (or
// recombines) an operand it does not use.
template <typename R, class Ld>
__device__ __forceinline__ void edge_operands(const Geo& g, Ld& ld, const C2<R>* __restrict__ Wx, int t, int xle,
                                              int xre, int lane, C2<R>& ep, C2<R>& ew) {
  ep = mk<R>(0, 0);
  ew = mk<R>(0, 0);
  if (lane < 2 * kMarchT) {
    const int rr = t + (lane < kMarchT ? lane : lane - kMarchT);
    ep = ld(rr * g.nx + (lane < kMarchT ? xle : xre));
    if (lane < kMarchT) ew = Wx[rr * g.nx + xle];
  }
}

// One warp marches rows ta .. tb-1 (tb > ta) of the 32 columns x0 = 32*xw ..
// x0+31, lane = column.  ld(i) yields the operand at site i (a plain load, or a
// vector recombined on the fly); epi(s, out(s), operand(s)) consumes each
// site's result.  psi(t-1), psi(t) and Wt(t-1) stay in registers from row to
// row; x neighbours come from warp shuffles.  Every load of a chunk of rows is
// issued before its first result is stored: the epilogue's stores may alias
// the operands as far as the compiler knows, and would otherwise hold each
// row's loads behind the previous row's stores, one memory latency per row.
template <int DAG, bool MU0, class Ld, class Epi>
__device__ __forceinline__ void march_segment32(const Geo& g, const OpK<float>& k, Ld& ld,
                                                const float2* __restrict__ Wt, const float2* __restrict__ Wx, int xw,
                                                int ta, int tb, Epi& epi) {
  using R = float;
  const int nx = g.nx;
  const int lane = threadIdx.x & 31;
  const Strip sp = strip_of(nx, xw, lane);
  const int last = sp.last, x = sp.x, xle = sp.xle, xre = sp.xre;
  const int tm = (ta == 0) ? g.nt - 1 : ta - 1;
  C2<R> pm = ld(tm * nx + x);
  C2<R> wtm = Wt[tm * nx + x];
  C2<R> pc = ld(ta * nx + x);
  int t = ta;
  for (; t + kMarchT <= tb; t += kMarchT) {
    C2<R> ep, ew;
    edge_operands<R>(g, ld, Wx, t, xle, xre, lane, ep, ew);
    C2<R> pp[kMarchT], wt[kMarchT], wx[kMarchT];
#pragma unroll
    for (int i = 0; i < kMarchT; i++) {
      const int tt = t + i;
      const int tp = (tt + 1 == g.nt) ? 0 : tt + 1;
      pp[i] = ld(tp * nx + x);
      wt[i] = Wt[tt * nx + x];
      wx[i] = Wx[tt * nx + x];
    }
#pragma unroll
    for (int i = 0; i < kMarchT; i++)
      march_row<R, DAG, MU0>(k, (t + i) * nx + x, lane, last, pm, pc, wtm, pp[i], wt[i], wx[i],
                             shfl_c2<R>(ep, (lane == last) ? kMarchT + i : i), shfl_c2<R>(ew, i), epi);
  }
  for (; t < tb; t++) {  // the last rows of the segment: lanes 0 and last fetch their own
    const int xe = (lane == last) ? xre : xle;
    const int tp = (t + 1 == g.nt) ? 0 : t + 1;
    const int s = t * nx + x;
    march_row<R, DAG, MU0>(k, s, lane, last, pm, pc, wtm, ld(tp * nx + x), Wt[s], Wx[s], ld(t * nx + xe), Wx[t * nx + xle],
                           epi);
  }
}

// Warp shuffles of block-floating operands and links (tg_fixed.cuh).
__device__ __forceinline__ FxC shfl_fx(const FxC& v, int src) {
  FxC o;
  o.re = __shfl_sync(0xffffffffu, v.re, src);
  o.im = __shfl_sync(0xffffffffu, v.im, src);
  o.e = __shfl_sync(0xffffffffu, v.e, src);
  return o;
}
__device__ __forceinline__ FxLink shfl_lk(FxLink w, int src) {
  return make_int4(__shfl_sync(0xffffffffu, w.x, src), __shfl_sync(0xffffffffu, w.y, src),
                   __shfl_sync(0xffffffffu, w.z, src), __shfl_sync(0xffffffffu, w.w, src));
}
__device__ __forceinline__ FxC sel_fx(bool c, const FxC& a, const FxC& b) {
  return FxC{c ? a.re : b.re, c ? a.im : b.im, c ? a.e : b.e};
}

// Rows whose loads are in flight together in the FP64 march.
constexpr int kChunk64 = 2;

// The FP64 march: march_segment32 with the operator on the integer pipes.  Each
// loaded operand is converted to block floating point once and shared with the
// neighbouring columns and rows in that form.
template <int DAG, bool MU0, class Ld, class Epi>
__device__ __forceinline__ void march_segment64(const Geo& g, const OpK<double>& k, Ld& ld,
                                                const FxLink* __restrict__ Wt, const FxLink* __restrict__ Wx, int xw,
                                                int ta, int tb, Epi& epi) {
  static_assert(kMarchT % kChunk64 == 0, "a chunk's edge operands are fetched kMarchT rows at a time");
  const int nx = g.nx;
  const int lane = threadIdx.x & 31;
  const Strip sp = strip_of(nx, xw, lane);
  const int last = sp.last, x = sp.x, xle = sp.xle, xre = sp.xre;
  const int tm = (ta == 0) ? g.nt - 1 : ta - 1;
  FxC pm = to_fx(ld(tm * nx + x));
  FxLink wtm = Wt[tm * nx + x];
  double2 own = ld(ta * nx + x);
  FxC pc = to_fx(own);
  // row t: in(t+1) = pp, in beyond the warp's edge pe (lanes 0 and last), the x link entering x0 we (lane 0)
  auto row = [&](int t, double2 pp, FxLink wt, FxLink wx, const FxC& pe, FxLink we) {
    const int s = t * nx + x;
    const FxC pr = sel_fx(lane == last, pe, shfl_fx(pc, lane + 1));
    const FxC pl = sel_fx(lane == 0, pe, shfl_fx(pc, lane - 1));
    FxLink wl = shfl_lk(wx, lane - 1);
    if (lane == 0) wl = we;
    const FxC pn = to_fx(pp);
    double2 o;
    if (!fx_dslash<DAG, MU0>(k, pc, pn, pm, pr, pl, wt, wtm, wx, wl, o)) {
      const Nbr n = neighbours(g, s, t, x);
      o = dslash_wide<DAG, MU0>(k, ld(s), ld(n.tp), ld(n.tm), ld(n.xp), ld(n.xm), wt, wtm, wx, wl);
    }
    if (lane <= last) epi(s, o, own);
    pm = pc;
    pc = pn;
    own = pp;
    wtm = wt;
  };
  int t = ta;
  for (; t + kMarchT <= tb; t += kMarchT) {
    // lane i < kMarchT: left of x0 in row t+i (and the link entering x0); lane kMarchT+i: right of x0+31
    double2 ep = make_double2(0, 0);
    FxLink ew = make_int4(0, 0, 0, 0);
    if (lane < 2 * kMarchT) {
      const int rr = t + (lane < kMarchT ? lane : lane - kMarchT);
      ep = ld(rr * nx + (lane < kMarchT ? xle : xre));
      if (lane < kMarchT) ew = Wx[rr * nx + xle];
    }
    const FxC ef = to_fx(ep);
#pragma unroll
    for (int h = 0; h < kMarchT; h += kChunk64) {
      double2 pp[kChunk64];
      FxLink wt[kChunk64], wx[kChunk64];
#pragma unroll
      for (int i = 0; i < kChunk64; i++) {
        const int tt = t + h + i;
        const int tp = (tt + 1 == g.nt) ? 0 : tt + 1;
        pp[i] = ld(tp * nx + x);
        wt[i] = Wt[tt * nx + x];
        wx[i] = Wx[tt * nx + x];
      }
#pragma unroll
      for (int i = 0; i < kChunk64; i++)
        row(t + h + i, pp[i], wt[i], wx[i], shfl_fx(ef, (lane == last) ? kMarchT + h + i : h + i), shfl_lk(ew, h + i));
    }
  }
  for (; t < tb; t++) {
    const int tp = (t + 1 == g.nt) ? 0 : t + 1;
    row(t, ld(tp * nx + x), Wt[t * nx + x], Wx[t * nx + x], to_fx(ld(t * nx + ((lane == last) ? xre : xle))),
        Wx[t * nx + xle]);
  }
}

// ---------------------------------------------------------------------------
// The FP64 march with its rows prefetched through shared memory: each lane copies
// its own column of the next rows -- the operand's sources, the links and the
// vectors the epilogue reads -- with cp.async (16 bytes, through L2), D rows
// ahead, and reads back only what it copied itself, so no barrier is needed.
// Prefetched rows cost no registers, and the epilogue's reads no longer wait
// behind the operator.  The edge operands of kMarchT rows are fetched likewise
// by the first lanes.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Shared memory per warp: D rows of NS + 2 + NE arrays, two chunks of edges.
template <int D, int NS, int NE> __host__ __device__ constexpr int ring_bytes() {
  return D * (NS + 2 + NE) * 512 + 2 * (NS + 1) * 2 * kMarchT * 16;
}

// The index arithmetic, host-callable for its audit: the row above row t; the slots of
// a march's row i and of its chunk's edges; the site of the edge operand that lane
// < 2 kMarchT fetches with the chunk whose first row is t (rows up to tb).
TG_HD int row_above(int nt, int t) { return t + 1 == nt ? 0 : t + 1; }
TG_HD int ring_slot(int i) { return i & (kMarchT - 1); }
TG_HD int ring_edge_slot(int i) { return (i / kMarchT) & 1; }
TG_HD int ring_edge(int nx, const Strip& p, int t, int tb, int lane) {
  return imin(t + (lane & (kMarchT - 1)), tb - 1) * nx + (lane < kMarchT ? p.xle : p.xre);
}

// src[NS]: the operand's sources (comb(v) gives the operand from their values at
// a site); ext[NE]: what the epilogue reads, handed to epi(s, out, operand, e).
template <int DAG, bool MU0, int D, int NS, int NE, class Comb, class Epi>
__device__ __forceinline__ void march_ring64(const Geo& g, const OpK<double>& k, const double2* const (&src)[NS],
                                             const double2* const* ext, Comb comb, const FxLink* __restrict__ Wt,
                                             const FxLink* __restrict__ Wx, int xw, int ta, int tb, Epi& epi,
                                             unsigned char* ring) {
  constexpr int NA = NS + 2 + NE, EL = 2 * kMarchT;
  const int nx = g.nx, n = tb - ta;
  const int lane = threadIdx.x & 31;
  const Strip st = strip_of(nx, xw, lane);
  const int last = st.last, x = st.x;
  double2* const rows = reinterpret_cast<double2*>(ring) + lane;
  double2* const edges = reinterpret_cast<double2*>(ring + D * NA * 512) + (lane & (EL - 1));
  const unsigned rows_a = smem_addr(rows), edges_a = smem_addr(edges);
  // row ta + i into slot `slot`; with every kMarchT-th row the edges of its chunk
  auto issue = [&](int i, int slot) {
    const int t = ta + i;
    const unsigned d = rows_a + slot * (NA * 512);
    const int so = t * nx + x, sp = row_above(g.nt, t) * nx + x;
    if (lane <= last) {  // (the spare lanes' copies of one address took a ragged strip's warps 17% longer)
#pragma unroll
      for (int j = 0; j < NS; j++) cp_async16(d + j * 512, src[j] + sp);
      cp_async16(d + NS * 512, Wt + so);
      cp_async16(d + (NS + 1) * 512, Wx + so);
#pragma unroll
      for (int j = 0; j < NE; j++) cp_async16(d + (NS + 2 + j) * 512, ext[j] + so);
    }
    if ((i & (kMarchT - 1)) == 0 && lane < EL) {
      const int c = ring_edge(nx, st, t, tb, lane);
      const unsigned e = edges_a + ring_edge_slot(i) * ((NS + 1) * EL * 16);
#pragma unroll
      for (int j = 0; j < NS; j++) cp_async16(e + j * (EL * 16), src[j] + c);
      if (lane < kMarchT) cp_async16(e + NS * (EL * 16), Wx + c);
    }
  };
#pragma unroll
  for (int i = 0; i < D - 1; i++) {
    if (i < n) issue(i, i);
    cp_async_commit();
  }
  auto at = [&](int s) {
    double2 v[NS];
#pragma unroll
    for (int j = 0; j < NS; j++) v[j] = __ldcg(src[j] + s);
    return comb(v);
  };
  const int tm = (ta == 0) ? g.nt - 1 : ta - 1;
  const double2 below = at(tm * nx + x);
  double2 own = at(ta * nx + x);
  FxLink wtm = Wt[tm * nx + x];
  FxC pm = to_fx(below), pc = to_fx(own), ef;
  FxLink ew;
  static_assert(D == kMarchT, "a chunk's rows and slots coincide");
  for (int i0 = 0; i0 < n; i0 += kMarchT) {
#pragma unroll
    for (int ic = 0; ic < kMarchT; ic++) {
      const int i = i0 + ic;
      if (i >= n) break;
      if (i + D - 1 < n) issue(i + D - 1, ring_slot(ic + D - 1));  // (i0 is a multiple of D)
      cp_async_commit();
      cp_async_wait<D - 1>();
      if (ic == 0) {
        const double2* e = edges + ring_edge_slot(i0) * ((NS + 1) * EL);
        double2 v[NS];
#pragma unroll
        for (int j = 0; j < NS; j++) v[j] = e[j * EL];
        ef = to_fx(comb(v));
        ew = *reinterpret_cast<const FxLink*>(e + NS * EL);
      }
      const double2* rw = rows + ic * (NA * 32);
      double2 v[NS];
#pragma unroll
      for (int j = 0; j < NS; j++) v[j] = rw[j * 32];
      const FxLink wt = *reinterpret_cast<const FxLink*>(rw + NS * 32);
      const FxLink wx = *reinterpret_cast<const FxLink*>(rw + (NS + 1) * 32);
      const double2 pp = comb(v);
      // the x neighbours and the link from x - 1, out of the lanes beside this one
      auto beside = [&](FxC& pr, FxC& pl, FxLink& wl) {
        const FxC pe = shfl_fx(ef, (lane == last) ? kMarchT + ic : ic);
        pr = sel_fx(lane == last, pe, shfl_fx(pc, lane + 1));
        pl = sel_fx(lane == 0, pe, shfl_fx(pc, lane - 1));
        const FxLink we = shfl_lk(ew, ic);
        wl = shfl_lk(wx, lane - 1);
        if (lane == 0) wl = we;
      };
      FxC pr, pl;
      FxLink wl;
      beside(pr, pl, wl);
      const FxC pn = to_fx(pp);
      const int t = ta + i, s = t * nx + x;
      double2 o;
      // (what the lanes beyond the strip's last hold is arbitrary, and of no use)
      const bool ok = fx_dslash<DAG, MU0>(k, pc, pn, pm, pr, pl, wt, wtm, wx, wl, o) || lane > last;
      // A vector that is zero in places has whole rows of refused sites, which are not worth
      // a reload and the FP64 form (1024^2 iteration on a point source 58 us, 192 with it).
      // The whole warp comes here, so that the neighbours can be shuffled again
      // instead of being kept in registers past the operator (a dense solve 52 us so, 53 kept).
      if (__any_sync(0xffffffffu, !ok)) {
        beside(pr, pl, wl);
        if (!ok) {
          if (fx_zero(pc) && fx_zero(pn) && fx_zero(pm) && fx_zero(pr) && fx_zero(pl) && fx_finite(k, wt, wtm, wx, wl)) {
            o = make_double2(0.0, 0.0);
          } else {
            const Nbr nb = neighbours(g, s, t, x);
            o = dslash_vals<double, DAG, MU0>(k, own, at(nb.tp), at(nb.tm), at(nb.xp), at(nb.xm), fx_link_value(wt),
                                              fx_link_value(wtm), fx_link_value(wx), fx_link_value(wl));
          }
        }
      }
      if (lane <= last) epi(s, o, own, rw + (NS + 2) * 32);
      pm = pc;
      pc = pn;
      own = pp;
      wtm = wt;
    }
  }
  cp_async_wait<0>();  // (only empty groups are left; the ring is free for the next segment)
}

template <typename R, int DAG, bool MU0, class Ld, class Epi>
__device__ __forceinline__ void march_segment(const Geo& g, const OpK<R>& k, Ld& ld, const Lk<R>* __restrict__ Wt,
                                              const Lk<R>* __restrict__ Wx, int xw, int ta, int tb, Epi& epi) {
  if constexpr (sizeof(R) == 4) march_segment32<DAG, MU0>(g, k, ld, Wt, Wx, xw, ta, tb, epi);
  else march_segment64<DAG, MU0>(g, k, ld, Wt, Wx, xw, ta, tb, epi);
}

// The (strip, t) rows of the lattice in strip-major order, split into one
// contiguous range per warp: ranges differ by at most one row, and a warp
// restarts its march only where its range crosses into a new strip.  Calls
// f(xw, ta, tb) for each strip segment of this warp's range.
template <class F> __device__ __forceinline__ void for_warp_rows(const Geo& g, F&& f) {
  const int wpb = (int)(blockDim.x >> 5);
  const long long rows = (long long)march_strips(g.nx) * g.nt;
  const long long nw = (long long)gridDim.x * wpb;
  const long long gw = (long long)blockIdx.x * wpb + (threadIdx.x >> 5);
  long long r = rows * gw / nw;
  const long long r1 = rows * (gw + 1) / nw;
  while (r < r1) {
    const int xw = (int)(r / g.nt);
    const int ta = (int)(r - (long long)xw * g.nt);
    const int tb = (r1 - r < (long long)(g.nt - ta)) ? ta + (int)(r1 - r) : g.nt;
    f(xw, ta, tb);
    r += tb - ta;
  }
}

// Apply the operator to every site and hand each result to epi: column march
// where the lattice allows it, else one site per thread.
template <typename R, int DAG, bool MU0, class Ld, class Epi>
__device__ __forceinline__ void stencil_ld(const Geo& g, const OpK<R>& k, Ld& ld, const Lk<R>* __restrict__ Wt,
                                           const Lk<R>* __restrict__ Wx, Epi& epi) {
  if (g.march) {
    for_warp_rows(g, [&](int xw, int ta, int tb) { march_segment<R, DAG, MU0>(g, k, ld, Wt, Wx, xw, ta, tb, epi); });
  } else {
    TG_SITES(s, g.V) {
      int t, x;
      site_tx(g, s, t, x);
      C2<R> own;
      const C2<R> o = dslash_ld<R, DAG, MU0>(g, k, ld, Wt, Wx, s, t, x, own);
      epi(s, o, own);
    }
  }
}

template <typename R, int DAG, bool MU0, class Epi>
__device__ __forceinline__ void stencil_all(const Geo& g, const OpK<R>& k, const C2<R>* __restrict__ in,
                                            const Lk<R>* __restrict__ Wt, const Lk<R>* __restrict__ Wx, Epi& epi) {
  auto ld = [&](int i) { return in[i]; };
  stencil_ld<R, DAG, MU0>(g, k, ld, Wt, Wx, epi);
}

// The operator over one small lattice run by a team of thread blocks (the
// batched-chain kernel: one block, or the blocks of a cluster).  T gives the
// block's rank in the team and the team's size.  The team's warps split the
// lattice's (strip, t) rows into one contiguous range each, as for_warp_rows
// splits them over a grid; lattices that do not march go one site per thread.
template <class T, typename R, int DAG, bool MU0, class Ld, class Epi>
__device__ __forceinline__ void stencil_team(const Geo& g, const OpK<R>& k, Ld& ld, const Lk<R>* __restrict__ Wt,
                                             const Lk<R>* __restrict__ Wx, Epi& epi) {
  const int wpb = blockDim.x >> 5;
  if (march_ok(g.nx)) {
    const int nw = T::nblocks() * wpb, w = T::rank() * wpb + (threadIdx.x >> 5);
    const int rows = march_strips(g.nx) * g.nt;
    int r = (int)((long long)rows * w / nw);
    const int r1 = (int)((long long)rows * (w + 1) / nw);
    while (r < r1) {
      const int xw = r / g.nt;
      const int ta = r - xw * g.nt;
      const int tb = (r1 - r < g.nt - ta) ? ta + (r1 - r) : g.nt;
      march_segment<R, DAG, MU0>(g, k, ld, Wt, Wx, xw, ta, tb, epi);
      r += tb - ta;
    }
  } else {
    for (int s = T::rank() * (int)blockDim.x + (int)threadIdx.x; s < g.V; s += T::nblocks() * (int)blockDim.x) {
      int t, x;
      site_tx(g, s, t, x);
      C2<R> own;
      const C2<R> o = dslash_ld<R, DAG, MU0>(g, k, ld, Wt, Wx, s, t, x, own);
      epi(s, o, own);
    }
  }
}

// ---------------------------------------------------------------------------
// TMA-staged march.  Each warp owns kStages stage buffers in dynamic shared
// memory, each holding one chunk (kMarchT rows) of its 32 columns: the
// operand sources of rows t+1 .. t+kMarchT and Wt, Wx of rows t .. t+kMarchT-1.
// Lane 0 fills a stage with one 32-site row segment per array and row
// (cp.async.bulk, 16-byte aligned because x0 is a multiple of 32) and arms
// the stage's mbarrier with the byte count; the warp waits on the barrier's
// phase, computes the chunk from shared memory, and lane 0 refills the stage
// with the chunk kStages ahead.  The operand of a site is combine() of its
// NSRC source arrays (one: a plain vector; two: r + beta p of CG).
// ---------------------------------------------------------------------------
template <typename R> struct SrcOne {  // the operand is a[i]
  static constexpr int n = 1;
  const C2<R>* a;
  __device__ __forceinline__ const C2<R>* arr(int) const { return a; }
  __device__ __forceinline__ C2<R> combine(const C2<R>* v) const { return v[0]; }
  __device__ __forceinline__ C2<R> operator()(int i) const { return a[i]; }
};

template <typename R> struct SrcAxpy {  // the operand is r[i] + beta p[i] (the CG direction p')
  static constexpr int n = 2;
  const C2<R>* r;
  const C2<R>* p;
  R beta;
  __device__ __forceinline__ const C2<R>* arr(int j) const { return j ? p : r; }
  __device__ __forceinline__ C2<R> combine(const C2<R>* v) const {
    return mk<R>(fma(beta, v[1].x, v[0].x), fma(beta, v[1].y, v[0].y));
  }
  __device__ __forceinline__ C2<R> operator()(int i) const {
    const C2<R> rv = r[i], pv = p[i];
    return mk<R>(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
  }
};

template <int NSRC> struct StageShape {
  static constexpr int stages = NSRC == 1 ? 4 : 3;  // 12 rows ahead at most, 12 KB per warp in FP32
};
template <typename R, int NSRC> __host__ __device__ constexpr int stage_bytes() {
  return (NSRC + 2) * kMarchT * 32 * (int)sizeof(C2<R>);
}
// Dynamic shared memory of a staged kernel: every warp's stages, then their mbarriers.
template <typename R, int NSRC> __host__ __device__ constexpr int staged_smem_bytes() {
  return (kBlock / 32) * (StageShape<NSRC>::stages * stage_bytes<R, NSRC>() + StageShape<NSRC>::stages * 8);
}

// Waits on a stage's mbarrier are bounded: kStageWaitLimit polls of
// try_wait (each suspends for a hardware-chosen slice).  A wait that runs
// out counts in g_stage_faults and the chunk is computed from whatever the
// stage holds, so a fault shows as an error count and wrong numbers, never as
// a hung GPU.
constexpr int kStageWaitLimit = 1 << 22;
static __device__ unsigned g_stage_faults;


__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// generic-proxy accesses to shared memory before later TMA writes to it
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void stage_wait(unsigned long long* bar, unsigned parity) {
  for (int it = 0; it < kStageWaitLimit; it++)
    if (mbar_try_wait(bar, parity)) return;
  if ((threadIdx.x & 31) == 0) atomicAdd(&g_stage_faults, 1u);
}

template <typename R, int DAG, bool MU0, class Src, class Epi>
__device__ __forceinline__ void march_segment_staged(const Geo& g, const OpK<R>& k, const Src& src,
                                                     const C2<R>* __restrict__ Wt, const C2<R>* __restrict__ Wx,
                                                     int xw, int ta, int tb, Epi& epi, unsigned char* stage,
                                                     unsigned long long* bars, unsigned& phases) {
  constexpr int NS = StageShape<Src::n>::stages;
  constexpr int RB = 32 * (int)sizeof(C2<R>);  // one row segment of one array
  constexpr int SB = stage_bytes<R, Src::n>();
  const int nx = g.nx;
  const int lane = threadIdx.x & 31;
  const int x0 = xw << 5;
  const int x = x0 + lane;
  const int xle = (x0 == 0) ? nx - 1 : x0 - 1;
  const int xre = (x0 + 32 == nx) ? 0 : x0 + 32;
  const int nchunks = (tb - ta) / kMarchT;
  // lane 0: chunk c (rows ta + c*kMarchT ..) into stage c % NS
  auto issue = [&](int c) {
    const int sg = c % NS;
    unsigned char* base = stage + sg * SB;
    const int t = ta + c * kMarchT;
    mbar_expect_tx(bars + sg, (unsigned)SB);
#pragma unroll
    for (int i = 0; i < kMarchT; i++) {
      const int tp = (t + i + 1 == g.nt) ? 0 : t + i + 1;
#pragma unroll
      for (int j = 0; j < Src::n; j++)
        bulk_g2s(base + (j * kMarchT + i) * RB, src.arr(j) + (size_t)tp * nx + x0, RB, bars + sg);
      bulk_g2s(base + (Src::n * kMarchT + i) * RB, Wt + (size_t)(t + i) * nx + x0, RB, bars + sg);
      bulk_g2s(base + ((Src::n + 1) * kMarchT + i) * RB, Wx + (size_t)(t + i) * nx + x0, RB, bars + sg);
    }
  };
  if (lane == 0) {
    fence_proxy_async_smem();
    for (int c = 0; c < nchunks && c < NS; c++) issue(c);
  }
  const int tm = (ta == 0) ? g.nt - 1 : ta - 1;
  C2<R> pm = src(tm * nx + x);
  C2<R> wtm = Wt[tm * nx + x];
  C2<R> pc = src(ta * nx + x);
  int t = ta;
  for (int c = 0; c < nchunks; c++, t += kMarchT) {
    const int sg = c % NS;
    C2<R> ep, ew;
    edge_operands<R>(g, src, Wx, t, xle, xre, lane, ep, ew);
    stage_wait(bars + sg, (phases >> sg) & 1u);
    phases ^= 1u << sg;
    const C2<R>* sv = reinterpret_cast<const C2<R>*>(stage + sg * SB);
#pragma unroll
    for (int i = 0; i < kMarchT; i++) {
      C2<R> v[Src::n];
#pragma unroll
      for (int j = 0; j < Src::n; j++) v[j] = sv[(j * kMarchT + i) * 32 + lane];
      march_row<R, DAG, MU0>(k, (t + i) * nx + x, lane, 31, pm, pc, wtm, src.combine(v),
                                   sv[(Src::n * kMarchT + i) * 32 + lane], sv[((Src::n + 1) * kMarchT + i) * 32 + lane],
                                   shfl_c2<R>(ep, (lane == 31) ? kMarchT + i : i), shfl_c2<R>(ew, i), epi);
    }
    __syncwarp();
    if (lane == 0 && c + NS < nchunks) {
      fence_proxy_async_smem();
      issue(c + NS);
    }
  }
  for (; t < tb; t++) {
    const int tp = (t + 1 == g.nt) ? 0 : t + 1;
    const int s = t * nx + x;
    const int xe = (lane == 31) ? xre : xle;
    march_row<R, DAG, MU0>(k, s, lane, 31, pm, pc, wtm, src(tp * nx + x), Wt[s], Wx[s], src(t * nx + xe),
                                 Wx[t * nx + xle], epi);
  }
}

// stencil_ld with the operand from Src, staged through shared memory on
// marching lattices.  The kernel must be launched with
// staged_smem_bytes<R, Src::n>() of dynamic shared memory.
template <typename R, int DAG, bool MU0, class Src, class Epi>
__device__ __forceinline__ void stencil_staged(const Geo& g, const OpK<R>& k, const Src& src,
                                               const C2<R>* __restrict__ Wt, const C2<R>* __restrict__ Wx, Epi& epi) {
  if (!g.march) {
    Src ld = src;
    stencil_ld<R, DAG, MU0>(g, k, ld, Wt, Wx, epi);
    return;
  }
  extern __shared__ __align__(128) unsigned char tg_dyn_smem[];
  constexpr int NS = StageShape<Src::n>::stages;
  constexpr int WB = NS * stage_bytes<R, Src::n>();
  const int w = threadIdx.x >> 5;
  unsigned char* stage = tg_dyn_smem + w * WB;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(tg_dyn_smem + (kBlock / 32) * WB) + w * NS;
  if ((threadIdx.x & 31) == 0) {
    for (int sg = 0; sg < NS; sg++) mbar_init(bars + sg, 1);
    mbar_init_fence();
  }
  __syncwarp();
  unsigned phases = 0;
  for_warp_rows(g, [&](int xw, int ta, int tb) {
    march_segment_staged<R, DAG, MU0>(g, k, src, Wt, Wx, xw, ta, tb, epi, stage, bars, phases);
  });
}

}  // namespace tg
