// tg_grid_cg.cu -- CG on M^dag M for middle-sized lattices, on chip: the grid's
// blocks (one per SM, cooperative) keep the whole solve in their shared memory.
//
// Between the cluster solver's lattices (tg_cluster_cg.cu) and those that no longer
// fit, an iteration of the grid solver (tg_pcg.cu) is mostly the latency of its
// loads: every pass begins with vectors and links from L2.  Here they stay on chip
// as in the cluster solver (tg_onchip.cuh).  What neighbouring blocks need -- the
// sites within nx of a block's ends -- goes through global memory, ordered by the
// grid barrier that the pass's sum needs anyway, and is read back into the window
// while the scalar warp adds the blocks' partials and computes alpha or beta.  Sums
// are integer sums (tg_scalar.cuh), taken again in FP64 where their scale does
// not fit.  Recurrences, stopping and reliable-update rules are tg_pcg.cu's.
//
// Bound: two grid barriers and sums, about 2.5 us of the 6.3 us at 128^2; above,
// the window's upkeep (at 256^2 a block keeps 431 sites and 512 neighbours) and the
// operator's integer instructions.  us per iteration before and after: FP64 128^2 9.3 -> 6.8, 256^2
// 12.1 -> 9.1, 400^2 19.9 -> 13.7; mixed 256^2 7.2 -> 5.8, 512^2 10.4 -> 7.8, 700^2 13.7 -> 9.8.
// Mixed lattices whose links no longer fit keep p, M p and r on chip and stream the
// links from L2, ahead of their use: 800^2 15.1 -> 12.0, 1000^2 19.5 -> 15.3, 1024^2 18.9 -> 16.1.
//
// The barrier's wait is bounded as in tg_pcg.cu: a block that gives up ends the solve with
// TG_E_TIMEOUT, and every other one times out at its next barrier.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "tg_gridbar.cuh"
#include "tg_onchip.cuh"

namespace tg {

constexpr int kGcgMaxBlocks = 512;

// One block's view of the exchange between passes.  All threads call its methods;
// T site threads come first, then the scalar warp.
struct GcgExchange {
  GridBar bar;
  longlong2* warp_part;  // shared: one per site warp
  int* fail;             // shared
  int T;

  // A grid barrier that follows the block's global stores.  prep() runs in the
  // scalar warp before its arrival (all lanes), after the block's own stores.
  template <class Prep> __device__ __forceinline__ void barrier(Prep prep) const {
    __syncthreads();
    if ((int)threadIdx.x >= T) {
      prep();
      if (!warp0_grid_wait(bar, gridDim.x, kBarrierSpinLimit) && threadIdx.x == T) *fail = 1;
    }
    __syncthreads();
  }
  __device__ __forceinline__ void barrier() const {
    barrier([] {});
  }
  // the same with the site threads' integer partials of v: the block's goes to
  // part[block] before the arrival
  template <typename R> __device__ __forceinline__ void post(R v, int ref, longlong2* part) const {
    if ((int)threadIdx.x < T) {
      const longlong2 q = fx_warp_partial(fx_term(v, ref));
      if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = q;
    }
    barrier([&] {
      const int lane = threadIdx.x & 31;
      const longlong2 q = lane < (T >> 5) ? warp_part[lane] : make_longlong2(0, 0);
      const unsigned low = __reduce_add_sync(0xffffffffu, (unsigned)q.x & 0x3ffffffu),
                     mid = __reduce_add_sync(0xffffffffu, (unsigned)(q.x >> 26) & 0x3ffffffu),
                     top = __reduce_add_sync(0xffffffffu, (unsigned)(q.x >> 52) + (unsigned)q.y);
      const unsigned long long lo = low + ((unsigned long long)mid << 26);
      // (one refused warp refuses the block; kGcgMaxBlocks of them fit 32 bits)
      if (lane == 0)
        part[blockIdx.x] = make_longlong2((long long)(lo & ((1ull << 52) - 1)),
                                          (long long)min(top + (unsigned)(lo >> 52), kFxTopRefused));
    });
  }
  // the grid's total of the blocks' partials, in the scalar warp
  __device__ __forceinline__ bool total(const longlong2* part, int ref, double& t) const {
    const int lane = threadIdx.x & 31, nb = (int)gridDim.x;
    longlong2 s = make_longlong2(0, 0);
    for (int j0 = 0; j0 < nb; j0 += 160) {
      longlong2 w[5];
#pragma unroll
      for (int j = 0; j < 5; j++) {
        const int i = j0 + lane + 32 * j;
        w[j] = i < nb ? __ldcg(part + i) : make_longlong2(0, 0);
      }
#pragma unroll
      for (int j = 0; j < 5; j++) {
        s.x += w[j].x;
        s.y += w[j].y;
      }
    }
    const unsigned low = __reduce_add_sync(0xffffffffu, (unsigned)s.x & 0x3ffffffu),
                   mid = __reduce_add_sync(0xffffffffu, (unsigned)(s.x >> 26) & 0x3ffffffu),
                   top = __reduce_add_sync(0xffffffffu, (unsigned)(s.x >> 52) + (unsigned)s.y);
    return fx_total_value(low, mid, top, ref, t);
  }
  // a sum in FP64 (fixed order), the same in every thread; part: one double per
  // block, not the one of the sum before it
  __device__ __forceinline__ double sum64(double v, double* part) const {
    __shared__ double sh[kCcgThreads / 32 + 1];
    __shared__ double s_out;
    v = ccg_warp_allsum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    barrier([&] {
      const int lane = threadIdx.x & 31;
      const double b = ccg_warp_allsum(lane <= (T >> 5) ? sh[lane] : 0.0);
      if (lane == 0) part[blockIdx.x] = b;
    });
    if ((int)threadIdx.x >= T) {
      double s = 0;
      for (int j = threadIdx.x & 31; j < (int)gridDim.x; j += 32) s += __ldcg(part + j);
      s = ccg_warp_allsum(s);
      if (threadIdx.x == T) s_out = s;
    }
    __syncthreads();
    return s_out;
  }
  // barrier among the site threads only
  __device__ __forceinline__ void sites_sync() const { asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory"); }
};

// f(window index, site) for this thread's share of the window's two halos
template <class F> __device__ __forceinline__ void gcg_halo(const CcgPart& P, int nx, int V, int T, F f) {
  for (int h = threadIdx.x; h < 2 * nx; h += T) {
    const int j = h < nx ? h : P.n + h;
    int s = P.b0 - nx + j;
    s += (s < 0) ? V : (s >= V ? -V : 0);
    f(j, s);
  }
}
__device__ __forceinline__ bool gcg_edge(const CcgPart& P, int nx, int i) { return i < nx || i >= P.n - nx; }

// FP64: the iteration of k_pcg64.  THREE: in 72 registers and at most 256 site threads, for
// lattices of which an SM holds three blocks (gcg_shape).
constexpr int kGcgThreeThreads = 256;
template <bool MU0, bool THREE>
__global__ void __launch_bounds__(THREE ? kGcgThreeThreads + 32 : kCcgThreads + 32, THREE ? 3 : 1)
k_gcg64(Pcg64Args a, int wmax, int nmax) {
  extern __shared__ __align__(16) unsigned char gcg_smem[];
  __shared__ CcgScalars sc;
  __shared__ longlong2 warp_part[kCcgThreads / 32];
  const Geo& g = a.g;
  const CcgPart P = ccg_part(g.V);
  const int nx = g.nx, n = P.n, win = n + 2 * nx, T = blockDim.x - 32, tid = threadIdx.x, nb = gridDim.x;
  const bool site = tid < T;  // else: the scalar warp
  const GcgExchange ex{a.bar, warp_part, &sc.fail, T};
  longlong2* const postA = reinterpret_cast<longlong2*>(a.part);
  longlong2* const postB = postA + nb;
  double* const part0 = a.part + 4 * nb;
  double* const part1 = a.part + 5 * nb;
  longlong2* pm = reinterpret_cast<longlong2*>(gcg_smem);
  longlong2* qm = pm + wmax;
  double2* p = reinterpret_cast<double2*>(qm + wmax);
  double2* r = p + wmax;
  FxLink* wt = reinterpret_cast<FxLink*>(r + wmax);
  FxLink* wx = wt + wmax;
  double2* x = reinterpret_cast<double2*>(wx + wmax);
  int* pe = reinterpret_cast<int*>(x + nmax);
  int* qe = pe + wmax;
  const FxArr pf{pm, pe}, qf{qm, qe};

  if (tid == T) {
    barrier_epoch() = 0;
    sc.fail = 0;
  }
  double v = 0;
  for (int j = tid; j < win; j += blockDim.x) {
    int s = P.b0 - nx + j;
    s += (s < 0) ? g.V : (s >= g.V ? -g.V : 0);
    const double2 bb = a.b[s];
    r[j] = bb;
    p[j] = bb;
    wt[j] = a.Wt[s];
    wx[j] = a.Wx[s];
    if (j >= nx && j < nx + n) {
      x[j - nx] = make_double2(0.0, 0.0);
      v = fma(bb.x, bb.x, v);
      v = fma(bb.y, bb.y, v);
    }
  }
  double rr = ex.sum64(v, part0);
  const double rr0 = rr, stop = ccg_stop(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  int status = -1, iter = 0, refA = fx_total_ref(rr0), refB = refA;
  if (sc.fail) status = TG_E_TIMEOUT;
  else if (isnan(rr)) status = TG_E_NAN;
  else if (!(rr >= stop) || rr == 0.0) status = TG_OK;
  auto tests = [&](double rn) { return cg_verdict(rn, stop, limit, iter + 1 >= a.maxiter); };
  int xp0, xm0;  // of the thread's first site
  ccg_x_offsets(g, min(P.b0 + tid, g.V - 1), xp0, xm0);
  auto offsets = [&](int i, int& xp, int& xm) {
    xp = xp0;
    xm = xm0;
    if (i != tid) ccg_x_offsets(g, P.b0 + i, xp, xm);
  };
  double beta = 0;
  while (status < 0) {
    double inv_rr = 0;
    if (site) {
      for (int j = tid; j < win; j += T) {
        const double2 rv = r[j], pv = p[j];
        const double2 pn = make_double2(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
        const FxC f = to_fx(pn);
        p[j] = pn;
        pm[j] = make_longlong2(f.re, f.im);
        pe[j] = f.e;
      }
      ex.sites_sync();
    } else {
      inv_rr = 1.0 / rr;
    }
    double va = 0;
    if (site)
      for (int i = tid; i < n; i += T) {
        int xp, xm;
        offsets(i, xp, xm);
        const double2 o = ccg_op64<0, MU0>(a.km, pf, wt, wx, nx + i, nx, xp, xm);
        const FxC f = to_fx(o);
        qm[nx + i] = make_longlong2(f.re, f.im);
        qe[nx + i] = f.e;
        if (gcg_edge(P, nx, i)) a.Mp[P.b0 + i] = o;
        va = fma(o.x, o.x, va);
        va = fma(o.y, o.y, va);
      }
    ex.post(va, refA, postA);
    auto apply = [&](int i) {
      int xp, xm;
      offsets(i, xp, xm);
      return ccg_op64<1, MU0>(a.kd, qf, wt, wx, nx + i, nx, xp, xm);
    };
    double2 ap = make_double2(0.0, 0.0);  // the thread's first site, before alpha is known
    if (site) {
      gcg_halo(P, nx, g.V, T, [&](int j, int s) {
        const FxC f = to_fx(__ldcg(a.Mp + s));
        qm[j] = make_longlong2(f.re, f.im);
        qe[j] = f.e;
      });
      ex.sites_sync();
      if (tid < n) ap = apply(tid);
    } else {
      double pap;
      const bool ok = ex.total(postA, refA, pap);
      if (tid == T) {
        sc.alpha = div_newton(rr, pap);
        sc.okA = ok;
        sc.refA = fx_total_ref(pap);
        sc.rr = rr;
      }
    }
    __syncthreads();
    double alpha = sc.alpha;
    refA = sc.refA;
    if (!sc.okA && !sc.fail) {
      const double pap = ex.sum64(va, part1);
      alpha = sc.rr / pap;
      refA = fx_total_ref(pap);
    }
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    double vb = 0;
    if (site)
      for (int i = tid; i < n; i += T) {
        if (i != tid) ap = apply(i);
        double2 xv = x[i], rv = r[nx + i];
        const double2 pv = p[nx + i];
        rv.x -= alpha * ap.x;
        rv.y -= alpha * ap.y;
        r[nx + i] = rv;
        if (gcg_edge(P, nx, i)) a.r[P.b0 + i] = rv;
        vb = fma(rv.x, rv.x, vb);
        vb = fma(rv.y, rv.y, vb);
        xv.x += alpha * pv.x;
        xv.y += alpha * pv.y;
        x[i] = xv;
      }
    ex.post(vb, refB, postB);
    if (site) {
      gcg_halo(P, nx, g.V, T, [&](int j, int s) { r[j] = __ldcg(a.r + s); });
    } else {
      double rn;
      const bool ok = ex.total(postB, refB, rn);
      if (tid == T) {
        sc.beta = div_prepared(rn, rr, inv_rr);
        sc.verdict = tests(rn);
        sc.okB = ok;
        sc.refB = fx_total_ref(rn);
        sc.rn = rn;
      }
    }
    __syncthreads();
    beta = sc.beta;
    status = sc.verdict;
    refB = sc.refB;
    double rn = sc.rn;
    if (!sc.okB && !sc.fail) {
      rn = ex.sum64(vb, part0);
      beta = rn / sc.rr;
      status = tests(rn);
      refB = fx_total_ref(rn);
    }
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    rr = rn;
    iter += 1;
  }
  for (int i = tid; i < n; i += blockDim.x) a.x[P.b0 + i] = x[i];
  ccg_report(a.st, a.log, a.log_index, rr, rr0, stop, iter, 0, status);
}

// Mixed: the iteration and the FP64 reliable update of k_pcgmx.  The FP64 x, its
// image M x and the FP64 links stay in global memory.  FORM:
//   kGcgSites   one site of a thread at a time
//   kGcgPairs   two sites of a row (nx is even), with half the loads: us per iteration
//               228^2 6.4 -> 6.1, 256^2 6.6 -> 6.1, 400^2 7.7 -> 7.3, 512^2 8.3 -> 7.8,
//               700^2 10.1 -> 9.8, 1000x200 7.5 -> 7.4, 50x1000 7.2 -> 6.7
//   kGcgStream  pairs, with the FP32 links and xs in global memory, for lattices of
//               which only p, M p and r fit; a thread has its next kGcgAhead pairs'
//               links in registers, at a pass's end those of the next pass.
//               Single sites, four ahead, took 18.3 us at 1000^2 (pairs: 15.3) and gained nothing
//               at 1024^2; 448, 416, 384 or 320 site threads 15.7, 15.6, 16.0, 17.1.
constexpr int kGcgSites = 0, kGcgStream = 1, kGcgPairs = 2, kGcgThree = 3;
constexpr int kGcgAhead = 2;
constexpr int kGcgStreamThreads = 480;  // with the scalar warp 16 warps: 128 registers instead of 96
struct GcgLinks {
  float4 t, td, x;  // of the pair: to t+1, from t-1, to x+1
  float2 xl;        // from x-1 into the first
};
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 pair_of(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float4& as4(float2* p) { return *reinterpret_cast<float4*>(p); }
__device__ __forceinline__ float4 as4(const float2* p) { return *reinterpret_cast<const float4*>(p); }

template <bool MU0, int FORM>
__global__ void __launch_bounds__(FORM == kGcgStream ? kGcgStreamThreads + 32 : kCcgThreads + 32, 1)
k_gcgmx(PcgMxArgs a, int wmax, int nmax) {
  extern __shared__ __align__(16) unsigned char gcg_smem[];
  __shared__ CcgScalars sc;
  __shared__ longlong2 warp_part[kCcgThreads / 32];
  const Geo& g = a.g;
  constexpr bool STREAM = FORM == kGcgStream, PAIRS = FORM != kGcgSites;
  CcgPart P = ccg_part(PAIRS ? g.V / 2 : g.V);
  if (PAIRS) {
    P.b0 *= 2;
    P.n *= 2;
  }
  const int nx = g.nx, n = P.n, win = n + 2 * nx, T = blockDim.x - 32, tid = threadIdx.x, nb = gridDim.x;
  const bool site = tid < T;  // else: the scalar warp
  const GcgExchange ex{a.bar, warp_part, &sc.fail, T};
  longlong2* const postA = reinterpret_cast<longlong2*>(a.part);
  longlong2* const postB = postA + nb;
  double* const part0 = a.part + 4 * nb;
  double* const part1 = a.part + 5 * nb;
  float2* p = reinterpret_cast<float2*>(gcg_smem);
  float2* q = p + wmax;
  float2* r = q + wmax;
  float2* wt = r + wmax;
  float2* wx = wt + wmax;
  float2* const xs = STREAM ? a.xs + P.b0 : wx + wmax;
  constexpr int U = STREAM ? kGcgAhead : 1;

  if (tid == T) {
    barrier_epoch() = 0;
    sc.fail = 0;
  }
  double v = 0;
  for (int j = tid; j < win; j += blockDim.x) {
    int s = P.b0 - nx + j;
    s += (s < 0) ? g.V : (s >= g.V ? -g.V : 0);
    const double2 bb = a.b[s];
    const float2 rb = make_float2((float)bb.x, (float)bb.y);
    r[j] = rb;
    p[j] = rb;
    if (!STREAM) {
      wt[j] = a.Wt32[s];
      wx[j] = a.Wx32[s];
    }
    if (j >= nx && j < nx + n) {
      if (!STREAM) xs[j - nx] = make_float2(0.f, 0.f);
      v = fma(bb.x, bb.x, v);
      v = fma(bb.y, bb.y, v);
    }
  }
  if (site)
    for (int i = tid; i < n; i += T) {
      a.x[P.b0 + i] = make_double2(0.0, 0.0);
      if (STREAM) xs[i] = make_float2(0.f, 0.f);
    }
  double rr = ex.sum64(v, part0);
  const double rr0 = rr, stop = ccg_stop(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  double drop = kRuDrop * rr;  // |r|^2 below which a reliable update is due
  int status = -1, iter = 0, n_ru = 0, since_ru = 0, refA = fx_total_ref(rr0), refB = refA;
  if (sc.fail) status = TG_E_TIMEOUT;
  else if (isnan(rr)) status = TG_E_NAN;
  else if (!(rr >= stop) || rr == 0.0) status = TG_OK;
  auto due = [&](double rn) -> int {  // a reliable update
    return since_ru + 1 >= a.ru_interval || iter + 1 >= a.maxiter || cg_update_due(rn, stop, drop, limit);
  };
  int xp0, xm0;  // of the thread's first site
  ccg_x_offsets(g, min(P.b0 + tid, g.V - 1), xp0, xm0);
  auto offsets = [&](int i, int& xp, int& xm) {
    xp = xp0;
    xm = xm0;
    if (i != tid) ccg_x_offsets(g, P.b0 + i, xp, xm);
  };
  // STREAM: the links of the pair at site i
  auto links = [&](int i) {
    const int s = P.b0 + i;
    int xp, xm;
    ccg_x_offsets(g, s, xp, xm);
    return GcgLinks{__ldg(reinterpret_cast<const float4*>(a.Wt32 + s)),
                    __ldg(reinterpret_cast<const float4*>(a.Wt32 + (s < nx ? s - nx + g.V : s - nx))),
                    __ldg(reinterpret_cast<const float4*>(a.Wx32 + s)), __ldg(a.Wx32 + s + xm)};
  };
  GcgLinks w[U];
  if (STREAM && site) {
#pragma unroll
    for (int u = 0; u < U; u++)
      if (2 * (tid + u * T) < n) w[u] = links(2 * (tid + u * T));
  }
  // f(i, u) for the thread's pairs; w[u] holds the links of the pair at i
  auto pairs = [&](auto f) {
    for (int i0 = 2 * tid; i0 < n; i0 += 2 * U * T) {
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + 2 * u * T;
        if (i < n) {
          f(i, u);
          if (STREAM) w[u] = links(i + 2 * U * T < n ? i + 2 * U * T : 2 * (tid + u * T));
        }
      }
    }
  };
  auto op2 = [&](auto dag, const OpK<float>& k, const float2* v, int i, int u) {
    int t, x;
    site_tx(g, P.b0 + i, t, x);
    const int j = nx + i, jl = x == 0 ? j + nx - 1 : j - 1, jr = x + 2 == nx ? j + 2 - nx : j + 2;
    const float4 c = as4(v + j), tu = as4(v + j + nx), td = as4(v + j - nx);
    const float2 left = v[jl], right = v[jr];
    const GcgLinks l = STREAM ? w[u] : GcgLinks{as4(wt + j), as4(wt + j - nx), as4(wx + j), wx[jl]};
    return pair_of(dslash_vals<float, decltype(dag)::value, MU0>(k, lo2(c), lo2(tu), lo2(td), hi2(c), left, lo2(l.t),
                                                                 lo2(l.td), lo2(l.x), l.xl),
                   dslash_vals<float, decltype(dag)::value, MU0>(k, hi2(c), hi2(tu), hi2(td), right, lo2(c), hi2(l.t),
                                                                 hi2(l.td), hi2(l.x), lo2(l.x)));
  };
  auto halo = [&](float2* v, const float2* src) {
    if constexpr (PAIRS) {
      for (int h = 2 * tid; h < 2 * nx; h += 2 * T) {
        const int j = h < nx ? h : n + h;
        int s = P.b0 - nx + j;
        s += (s < 0) ? g.V : (s >= g.V ? -g.V : 0);
        as4(v + j) = __ldcg(reinterpret_cast<const float4*>(src + s));
      }
    } else {
      gcg_halo(P, nx, g.V, T, [&](int j, int s) { v[j] = __ldcg(src + s); });
    }
  };
  float4 xa[U];  // STREAM: xs of the thread's next U pairs
  float bf = 0.f;
  while (status < 0) {
    double inv_rr = 0;
    if (site) {
      if constexpr (PAIRS) {
        for (int j = 2 * tid; j < win; j += 2 * T) {
          const float4 rv = as4(r + j), pv = as4(p + j);
          as4(p + j) = make_float4(fmaf(bf, pv.x, rv.x), fmaf(bf, pv.y, rv.y), fmaf(bf, pv.z, rv.z), fmaf(bf, pv.w, rv.w));
        }
      } else {
        for (int j = tid; j < win; j += T) {
          const float2 rv = r[j], pv = p[j];
          p[j] = make_float2(fmaf(bf, pv.x, rv.x), fmaf(bf, pv.y, rv.y));
        }
      }
      ex.sites_sync();
    } else {
      inv_rr = 1.0 / rr;
    }
    float va = 0;
    if (site) {
      if constexpr (PAIRS) {
        pairs([&](int i, int u) {
          const float4 o = op2(std::integral_constant<int, 0>{}, a.km32, p, i, u);
          va = fmaf(o.x, o.x, va);
          va = fmaf(o.y, o.y, va);
          va = fmaf(o.z, o.z, va);
          va = fmaf(o.w, o.w, va);
          as4(q + nx + i) = o;
          if (gcg_edge(P, nx, i)) as4(a.Mp + P.b0 + i) = o;
        });
#pragma unroll
        for (int u = 0; u < U; u++)
          if (STREAM && 2 * (tid + u * T) < n) xa[u] = as4(xs + 2 * (tid + u * T));
      } else {
        for (int i = tid; i < n; i += T) {
          int xp, xm;
          offsets(i, xp, xm);
          const float2 o = ccg_op32<0, MU0>(a.km32, p, wt, wx, nx + i, nx, xp, xm);
          va = fmaf(o.x, o.x, va);
          va = fmaf(o.y, o.y, va);
          q[nx + i] = o;
          if (gcg_edge(P, nx, i)) a.Mp[P.b0 + i] = o;
        }
      }
    }
    ex.post(va, refA, postA);
    auto apply = [&](int i) {
      int xp, xm;
      offsets(i, xp, xm);
      return ccg_op32<1, MU0>(a.kd32, q, wt, wx, nx + i, nx, xp, xm);
    };
    auto apply2 = [&](int i, int u) { return op2(std::integral_constant<int, 1>{}, a.kd32, q, i, u); };
    float4 ap2 = make_float4(0.f, 0.f, 0.f, 0.f);  // of the thread's first pair
    float2 ap = make_float2(0.f, 0.f);  // the thread's first site, before alpha is known
    if (site) {
      halo(q, a.Mp);
      ex.sites_sync();
      if constexpr (PAIRS) {
        if (2 * tid < n) ap2 = apply2(2 * tid, 0);
      } else if (tid < n) {
        ap = apply(tid);
      }
    } else {
      double pap;
      const bool ok = ex.total(postA, refA, pap);
      if (tid == T) {
        sc.af = (float)div_newton<false>(rr, pap);
        sc.okA = ok;
        sc.refA = fx_total_ref(pap);
        sc.rr = rr;
      }
    }
    __syncthreads();
    float af = sc.af;
    refA = sc.refA;
    if (!sc.okA && !sc.fail) {
      const double pap = ex.sum64((double)va, part1);
      af = (float)(sc.rr / pap);
      refA = fx_total_ref(pap);
    }
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    float vb = 0;
    if (site) {
      if constexpr (PAIRS) {
        pairs([&](int i, int u) {
          if (i != 2 * tid) ap2 = apply2(i, u);
          float4 xv = STREAM ? xa[u] : as4(xs + i), rv = as4(r + nx + i);
          const float4 pv = as4(p + nx + i);
          rv.x = fmaf(-af, ap2.x, rv.x);
          rv.y = fmaf(-af, ap2.y, rv.y);
          rv.z = fmaf(-af, ap2.z, rv.z);
          rv.w = fmaf(-af, ap2.w, rv.w);
          as4(r + nx + i) = rv;
          if (gcg_edge(P, nx, i)) as4(a.r + P.b0 + i) = rv;
          vb = fmaf(rv.x, rv.x, vb);
          vb = fmaf(rv.y, rv.y, vb);
          vb = fmaf(rv.z, rv.z, vb);
          vb = fmaf(rv.w, rv.w, vb);
          xv.x = fmaf(af, pv.x, xv.x);
          xv.y = fmaf(af, pv.y, xv.y);
          xv.z = fmaf(af, pv.z, xv.z);
          xv.w = fmaf(af, pv.w, xv.w);
          as4(xs + i) = xv;
          if (STREAM && i + 2 * U * T < n) xa[u] = as4(xs + i + 2 * U * T);
        });
      } else {
        for (int i = tid; i < n; i += T) {
          if (i != tid) ap = apply(i);
          float2 xv = xs[i], rv = r[nx + i];
          const float2 pv = p[nx + i];
          rv.x = fmaf(-af, ap.x, rv.x);
          rv.y = fmaf(-af, ap.y, rv.y);
          r[nx + i] = rv;
          if (gcg_edge(P, nx, i)) a.r[P.b0 + i] = rv;
          vb = fmaf(rv.x, rv.x, vb);
          vb = fmaf(rv.y, rv.y, vb);
          xv.x = fmaf(af, pv.x, xv.x);
          xv.y = fmaf(af, pv.y, xv.y);
          xs[i] = xv;
        }
      }
    }
    ex.post(vb, refB, postB);
    if (site) {
      halo(r, a.r);
    } else {
      double rn;
      const bool ok = ex.total(postB, refB, rn);
      if (tid == T) {
        sc.bf = (float)(rn * inv_rr);
        sc.verdict = due(rn);
        sc.okB = ok;
        sc.refB = fx_total_ref(rn);
        sc.rn = rn;
      }
    }
    __syncthreads();
    bf = sc.bf;
    refB = sc.refB;
    int need = sc.verdict;
    double rn = sc.rn;
    if (!sc.okB && !sc.fail) {
      rn = ex.sum64((double)vb, part0);
      bf = (float)(rn / sc.rr);
      need = due(rn);
      refB = fx_total_ref(rn);
    }
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    rr = rn;
    iter += 1;
    since_ru += 1;
    if (!need) continue;
    // reliable update: x += xs, xs = 0; r = b - M^dag M x in FP64; r32 = (float) r
    if (site)
      for (int i = tid; i < n; i += T) {
        const float2 d = xs[i];
        double2 xv = __ldcg(a.x + P.b0 + i);
        xv.x += (double)d.x;
        xv.y += (double)d.y;
        a.x[P.b0 + i] = xv;
        xs[i] = make_float2(0.f, 0.f);
      }
    ex.barrier();
    auto ld_x = [&](int s) { return __ldcg(a.x + s); };
    if (site)
      for (int i = tid; i < n; i += T) {
        int t, xx;
        double2 own;
        site_tx(g, P.b0 + i, t, xx);
        a.tmp[P.b0 + i] = dslash_ld<double, 0, MU0>(g, a.km, ld_x, a.Wt, a.Wx, P.b0 + i, t, xx, own);
      }
    ex.barrier();
    double vt = 0;
    auto ld_t = [&](int s) { return __ldcg(a.tmp + s); };
    if (site)
      for (int i = tid; i < n; i += T) {
        int t, xx;
        double2 own;
        const int s = P.b0 + i;
        site_tx(g, s, t, xx);
        const double2 ap64 = dslash_ld<double, 1, MU0>(g, a.kd, ld_t, a.Wt, a.Wx, s, t, xx, own), bb = a.b[s];
        const double2 rv = make_double2(bb.x - ap64.x, bb.y - ap64.y);
        const float2 r32 = make_float2((float)rv.x, (float)rv.y);
        r[nx + i] = r32;
        if (gcg_edge(P, nx, i)) a.r[s] = r32;
        vt = fma(rv.x, rv.x, vt);
        vt = fma(rv.y, rv.y, vt);
      }
    const double rt = ex.sum64(vt, part1);
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    if (site) halo(r, a.r);
    __syncthreads();
    if (rt > kRuRestart * rr) bf = 0.f;  // the recursive residual was far too optimistic: restart p from r
    drop = kRuDrop * rt;
    rr = rt;
    since_ru = 0;
    n_ru += 1;
    if (isnan(rt)) status = TG_E_NAN;
    else if (rt < stop) status = TG_OK;
    else if (rt > limit) status = TG_E_DIVERGED;
    else if (iter >= a.maxiter) status = TG_E_NOCONV;
  }
  ccg_report(a.st, a.log, a.log_index, rr, rr0, stop, iter, n_ru, status);
}

// ---------------------------------------------------------------------------
// Launch
// ---------------------------------------------------------------------------
// sites of the largest block
static int gcg_most_sites(int V, int nblocks, int form) {
  return form == kGcgPairs || form == kGcgStream ? (V / 2 + nblocks - 1) / nblocks * 2 : (V + nblocks - 1) / nblocks;
}
static size_t gcg_bytes(const Geo& g, int nblocks, bool mixed, int form) {
  const size_t nmax = gcg_most_sites(g.V, nblocks, form), win = nmax + 2 * (size_t)g.nx;
  if (form == kGcgStream) return win * 3 * sizeof(float2);
  return win * (mixed ? kCcg32Window : kCcg64Window) + nmax * (mixed ? kCcg32Own : kCcg64Own);
}

// blocks that are resident at once on the current device (one per SM), 0 if the
// kernels cannot run
static int gcg_resident() {
  static std::mutex mu;
  static std::unordered_map<int, int> cache;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(dev);
  if (it != cache.end()) return it->second;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 0;
  const struct {
    const void* k;
    int threads;
  } kernels[] = {{(const void*)k_gcg64<true, false>, kCcgThreads},
                 {(const void*)k_gcg64<false, false>, kCcgThreads},
                 {(const void*)k_gcg64<true, true>, kGcgThreeThreads},
                 {(const void*)k_gcg64<false, true>, kGcgThreeThreads},
                 {(const void*)k_gcgmx<true, kGcgSites>, kCcgThreads},
                 {(const void*)k_gcgmx<false, kGcgSites>, kCcgThreads},
                 {(const void*)k_gcgmx<true, kGcgPairs>, kCcgThreads},
                 {(const void*)k_gcgmx<false, kGcgPairs>, kCcgThreads},
                 {(const void*)k_gcgmx<true, kGcgStream>, kGcgStreamThreads},
                 {(const void*)k_gcgmx<false, kGcgStream>, kGcgStreamThreads}};
  for (const auto& q : kernels) {
    int n = 0;
    if (cudaFuncSetAttribute(q.k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCcgSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, q.k, q.threads + 32, kCcgSmem) != cudaSuccess || n < 1)
      sms = 0;
  }
  (void)cudaGetLastError();
  cache.emplace(dev, sms);
  return sms;
}

// Where it runs (us per iteration on GB300: this solver / the cluster solver / the
// grid solver of tg_pcg.cu, whose passes read everything from L2):
//   FP64   64^2 5.8 / 4.3 / 9.3   90^2 6.2 / 6.1 / 9.3   128^2 6.8 / - / 9.3
//          256^2 9.1 / - / 12.1   400^2 13.7 / - / 19.9  16x1000 8.9 / - / 9.3
//   mixed  128^2 5.6 / 4.1 / 6.3  190^2 6.0 / 5.3 / 6.5  228^2 6.0 / 6.8 / 7.0
//          256^2 5.8 / - / 7.2    512^2 7.8 / - / 10.4   700^2 9.8 / - / 13.7
// In FP64 a cluster of 16 blocks is faster while each of its threads has one site
// (512 a block), mixed up to 2400 sites a block.  Beyond, this solver takes what its
// shared memory holds: about 170 000 sites in FP64 and 650 000 mixed, less the
// window; mixed lattices of even rows up to about 1.1 million sites stream their links
// (this solver / the grid solver: 600x1300 14.0 / 17.3, 3000x300 13.8 / 18.9, 10000x80 12.7 / 17.3,
// 250x2600 15.0 / 15.8, 1056x1040 16.7 / 20.1).  Mixed lattices whose rows span more than three blocks lose to the
// window's upkeep (40x1500 7.4 / - / 7.2, 20x2000 7.2 / - / 6.6; 50x1000 7.0 / - / 7.2).
// One block per SM: half of them cost 8.7 -> 11.3 at 256^2.  Threads: a site each, and
// no fewer than half the window (16x1000 12.0 -> 8.9 with 544 instead of 128).
//
// Several lattices at once, each on its own stream and thread, share the SMs: a lattice of up to
// a few hundred sites a block therefore takes no more threads and registers
// than let an SM hold the blocks of two to four (an SM's quarter holds 5 warps of 96 registers, 7 of
// 72).  us per iteration and lattice, 1 / 4 / 8 / 16 lattices, with the threads of one site each, and so:
//   FP64   128^2 6.4 / 3.6 / 3.5 / 3.5 -> 6.8 / 2.3 / 1.9 / 1.9    192^2 7.3 / 7.2 / 7.2 / 7.2 -> 7.6 / 3.4 / 3.4 / 3.3
//          256^2 8.9 / 8.8 / 8.8 / 8.8 -> 9.0 / 5.2 / 5.2 / 5.2    40x330 7.3 / 7.1 / 7.0 -> 7.1 / 3.9 / 3.8
//   mixed  256^2 6.2 / 3.2 / 3.2 / 3.2 -> 5.8 / 1.8 / 1.8 / 1.8    278^2 6.3 / 3.3 / 3.3 / 3.2 -> 6.3 / 1.9 / 1.9 / 1.9
// FP64, up to 256 sites a block where three fit the shared memory: the 72-register instance, a site a
// thread, and no fewer than a third of the window; up to 512 where two fit: 256 threads.  Mixed,
// up to 512 sites a block where four fit: two pairs a thread.
constexpr int kGcgSites64 = 512, kGcgSitesMx = 2400;
constexpr size_t kSmSmem = 228 * 1024, kBlockSmem = 1024 + 512;  // an SM's, and a block's besides its dynamic

CcgShape gcg_shape(const Geo& g, bool mixed, const CcgShape& cluster) {
  const CcgShape none{0, 0, 0};
  if (getenv("TG_PCG_BLOCK") != nullptr || getenv("TG_MIXED_CG") != nullptr) return none;
  const char *e = getenv("TG_GRID_CG"), *cl = getenv("TG_CLUSTER_CG");
  int want = 1 << 20, threads = 0, form = e ? kGcgSites : kGcgPairs;
  if (e && sscanf(e, "%d:%d:%d", &want, &threads, &form) >= 1 && want <= 0) return none;
  if (cluster.blocks > 0) {
    const int n = (g.V + cluster.blocks - 1) / cluster.blocks;
    if (cl || n <= (mixed ? kGcgSitesMx : kGcgSites64)) return none;
  } else if (!e && cl && cl[0] == '0') {
    return none;  // the on-chip solvers are turned off
  }
  const int sms = std::min(kGcgMaxBlocks, gcg_resident());
  if (sms <= 0) return none;
  const int blocks = std::max(1, std::min(std::min(want, sms), g.V / 64));
  const int n = (g.V + blocks - 1) / blocks;
  if (!mixed || (form == kGcgPairs && g.nx % 2 != 0)) form = kGcgSites;
  if (mixed && gcg_bytes(g, blocks, true, form) > (size_t)kCcgSmem) form = kGcgStream;
  if (form == kGcgStream && g.nx % 2 != 0) return none;
  if (gcg_bytes(g, blocks, mixed, form) > (size_t)kCcgSmem) return none;
  if (!e && mixed && g.nx > 3 * n) return none;
  auto fit = [&](size_t k) { return k * (gcg_bytes(g, blocks, mixed, form) + kBlockSmem) <= kSmSmem; };
  int t = threads > 0 ? threads : std::max(n, n / 2 + g.nx) / (form != kGcgSites ? 2 : 1), most = kCcgThreads;
  if (form == kGcgStream) {
    most = kGcgStreamThreads;
  } else if (!mixed && n <= 256 && (threads <= 0 || t <= kGcgThreeThreads) && fit(3)) {
    form = kGcgThree;
    most = kGcgThreeThreads;
    if (threads <= 0) t = std::max(n, (n + 2 * g.nx + 2) / 3);
  } else if (!mixed && threads <= 0 && n <= 512 && fit(2)) {
    most = 256;
  } else if (form == kGcgPairs && threads <= 0 && n <= 512 && fit(4)) {
    most = 128;
  }
  return CcgShape{blocks, std::min(most, (t + 31) / 32 * 32), form};
}

template <class K, class Args>
static cudaError_t gcg_launch(K kernel, cudaStream_t s, const Args& a, bool mixed, const CcgShape& sh) {
  const int nmax = gcg_most_sites(a.g.V, sh.blocks, sh.form);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sh.blocks);
  cfg.blockDim = dim3((unsigned)sh.threads + 32);  // and the scalar warp
  cfg.dynamicSmemBytes = gcg_bytes(a.g, sh.blocks, mixed, sh.form);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, a, nmax + 2 * a.g.nx, nmax);
}

cudaError_t gcg64(cudaStream_t s, bool mu0, const Pcg64Args& a, const CcgShape& sh) {
  if (sh.form == kGcgThree)
    return mu0 ? gcg_launch(k_gcg64<true, true>, s, a, false, sh) : gcg_launch(k_gcg64<false, true>, s, a, false, sh);
  return mu0 ? gcg_launch(k_gcg64<true, false>, s, a, false, sh) : gcg_launch(k_gcg64<false, false>, s, a, false, sh);
}
cudaError_t gcgmx(cudaStream_t s, bool mu0, const PcgMxArgs& a, const CcgShape& sh) {
  switch (sh.form) {
    case kGcgStream:
      return mu0 ? gcg_launch(k_gcgmx<true, kGcgStream>, s, a, true, sh) : gcg_launch(k_gcgmx<false, kGcgStream>, s, a, true, sh);
    case kGcgPairs:
      return mu0 ? gcg_launch(k_gcgmx<true, kGcgPairs>, s, a, true, sh) : gcg_launch(k_gcgmx<false, kGcgPairs>, s, a, true, sh);
    default:
      return mu0 ? gcg_launch(k_gcgmx<true, kGcgSites>, s, a, true, sh) : gcg_launch(k_gcgmx<false, kGcgSites>, s, a, true, sh);
  }
}

}  // namespace tg
