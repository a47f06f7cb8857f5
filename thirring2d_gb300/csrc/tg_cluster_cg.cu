// tg_cluster_cg.cu -- CG on M^dag M for small lattices, on chip: one
// thread-block cluster keeps the whole solve in its blocks' shared memory.
//
// A small lattice's CG iteration is bound by latency: on the grid-wide solver
// (tg_pcg.cu) each of its two sums is a grid barrier through L2 and a read of
// the partials (about 2 us), and each pass starts with loads from L2.  Here a
// block owns the sites [V c / N, V (c + 1) / N) of the t-major order, and keeps
// them and a window of nx sites on either side, which holds every neighbour of
// its own sites, in shared memory.  A pass reads shared memory only.  A value
// that a neighbouring block's window holds too is sent there as it is computed,
// and so is every warp's partial of the pass's sum to every block, by
// asynchronous stores into distributed shared memory (st.async) that count on
// the receiving block's mbarrier.  One wait on it per pass hands on the halo and
// the sum together, without a cluster barrier, whose release would wait for the
// remote stores to be acknowledged (measured 1100-1400 clocks a pass; the wait
// for the last block's sends 250-600).  p' = r + beta p is formed on the whole window by every block that
// holds it (the same operation on the same bits).
//
// The waits order the buffers' reuse too: a block sends into a window or partial
// array again only after it has received every warp's partial of the sum in
// between, which that warp sent after its reads.
//
// The recurrences, the stopping and reliable-update rules and the results are
// tg_pcg.cu's, up to the rounding of the sums.  Every block has all warps'
// partials, so all blocks take the same branches.
//
// What is left is latency (tg_scalar.cuh), so the scalar steps are kept off the
// sites' way: the last warp of a block has no sites.  It adds the partials and
// computes alpha while the others apply M^dag, and 1 / |r|^2, which beta needs,
// while they apply M.  The sums are integer sums; one whose scale does not fit
// is taken again in FP64 (ccg_sum).
#include <cooperative_groups.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "tg_onchip.cuh"

namespace tg {

namespace cg = cooperative_groups;

constexpr int kCcgMaxBlocks = 16;              // largest cluster
constexpr int kCcgPart = kCcgMaxBlocks * (kCcgThreads / 32 + 1);

template <typename T> __device__ __forceinline__ T* ccg_remote(T* p, int block) {
  return cg::this_cluster().map_shared_rank(p, (unsigned)block);
}

// Store v at own site i (window index nx + i) of arr, and in the windows of the
// neighbouring blocks that hold the site.  All blocks' arrays lie at the same
// shared addresses; a window is [nx below | own | nx above].  Plain stores, for
// the steps that end in a cluster barrier.
template <typename T> __device__ __forceinline__ void ccg_store(T* arr, const CcgPart& p, int nx, int i, T v) {
  arr[nx + i] = v;
  if (i < nx) ccg_remote(arr, p.prev)[nx + p.nprev + i] = v;
  if (i >= p.n - nx) ccg_remote(arr, p.next)[i - (p.n - nx)] = v;
}

// ---------------------------------------------------------------------------
// Asynchronous stores to a block of the cluster, counted on its mbarrier.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned ccg_smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned ccg_map(unsigned addr, int block) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(block));
  return r;
}
__device__ __forceinline__ void ccg_send(unsigned dst, unsigned bar, longlong2 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "l"(v.x), "l"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ccg_send(unsigned dst, unsigned bar, double2 v) {
  ccg_send(dst, bar, make_longlong2(__double_as_longlong(v.x), __double_as_longlong(v.y)));
}
__device__ __forceinline__ void ccg_send(unsigned dst, unsigned bar, float2 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ccg_send(unsigned dst, unsigned bar, int v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(v),
               "r"(bar)
               : "memory");
}
// as ccg_store, the neighbours' copies sent
template <typename T>
__device__ __forceinline__ void ccg_store_send(T* arr, const CcgPart& p, int nx, int i, T v, unsigned bar) {
  arr[nx + i] = v;
  if (i < nx) ccg_send(ccg_map(ccg_smem_addr(arr + nx + p.nprev + i), p.prev), ccg_map(bar, p.prev), v);
  if (i >= p.n - nx) ccg_send(ccg_map(ccg_smem_addr(arr + i - (p.n - nx)), p.next), ccg_map(bar, p.next), v);
}

// A pass's mbarrier: one arrival per site warp of the block (its own stores), one
// that announces the bytes to come, and those bytes.
__device__ __forceinline__ void ccg_bar_init(unsigned bar, int site_warps) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(site_warps + 1) : "memory");
}
__device__ __forceinline__ void ccg_bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ccg_bar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded: a thread that gives up sets *fail, which the block reads after its next
// block barrier.
__device__ __forceinline__ void ccg_bar_wait(unsigned bar, unsigned parity, int* fail) {
  unsigned done = 0;
  for (int i = 0; i < (1 << 16); i++) {  // each try may suspend the thread for some microseconds
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return;
  }
  *fail = 1;
}

// The cluster's total of the threads' partials in FP64 (fixed order), handed to
// f, which runs in thread 0 of every block; every thread gets f's result.  The
// cluster barrier also orders every store made before the call.  `part` holds
// one double per warp of the cluster; between two calls there is another
// cluster barrier, so that a block never writes one that is still being read.
template <class F>
__device__ __forceinline__ auto ccg_sum(double v, double* part, const CcgPart& p, F f) -> decltype(f(0.0)) {
  using S = decltype(f(0.0));
  __shared__ S s_out;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = ccg_warp_allsum(v);
  if (lane < p.nblocks) ccg_remote(part, lane)[p.c * nw + w] = v;
  cg::this_cluster().sync();
  if (w == 0) {
    double s = 0;
    for (int j = lane; j < p.nblocks * nw; j += 32) s += part[j];
    s = ccg_warp_allsum(s);
    if (lane == 0) s_out = f(s);
  }
  __syncthreads();
  return s_out;
}

// Every site warp's integer partial, into every block's array; and the warp's
// arrival, after its stores.
template <typename R>
__device__ __forceinline__ void ccg_post(R v, int ref, longlong2* part, const CcgPart& p, int nsw, unsigned bar) {
  const longlong2 q = fx_warp_partial(fx_term(v, ref));  // R: FP32 or FP64 terms
  const int lane = threadIdx.x & 31;
  if (lane < p.nblocks)
    ccg_send(ccg_map(ccg_smem_addr(part + p.c * nsw + (threadIdx.x >> 5)), lane), ccg_map(bar, lane), q);
  __syncwarp();
  if (lane == 0) ccg_bar_arrive(bar);
}

// The end of a kernel: no block leaves while another may still write into its
// shared memory.  After a wait that gave up the others may be up to five cluster
// barriers (two sums in FP64 and a reliable update) from giving up themselves.
__device__ __forceinline__ void ccg_leave(bool failed) {
  const int k = failed ? 8 : 1;
  for (int i = 0; i < k; i++) cg::this_cluster().sync();
}

// FP64: the iteration of k_pcg64
template <bool MU0> __global__ void __launch_bounds__(kCcgThreads + 32, 1) k_ccg64(Pcg64Args a, int wmax, int nmax) {
  extern __shared__ __align__(16) unsigned char ccg_smem[];
  __shared__ CcgScalars sc;
  __shared__ __align__(8) unsigned long long bars[2];
  const Geo& g = a.g;
  const CcgPart P = ccg_part(g.V);
  const int nx = g.nx, n = P.n, win = n + 2 * nx, T = blockDim.x - 32, tid = threadIdx.x, nsw = T >> 5;
  const bool site = tid < T;  // else: the scalar warp
  longlong2* postA = reinterpret_cast<longlong2*>(ccg_smem);
  longlong2* postB = postA + kCcgPart;
  double* part = reinterpret_cast<double*>(postB + kCcgPart);
  longlong2* pm = reinterpret_cast<longlong2*>(part + kCcgPart);
  longlong2* qm = pm + wmax;
  double2* p = reinterpret_cast<double2*>(qm + wmax);
  double2* r = p + wmax;
  FxLink* wt = reinterpret_cast<FxLink*>(r + wmax);
  FxLink* wx = wt + wmax;
  double2* x = reinterpret_cast<double2*>(wx + wmax);
  int* pe = reinterpret_cast<int*>(x + nmax);
  int* qe = pe + wmax;
  const FxArr pf{pm, pe}, qf{qm, qe};

  const unsigned barA = ccg_smem_addr(&bars[0]), barB = ccg_smem_addr(&bars[1]);
  const unsigned bytesA = P.nblocks * nsw * 16 + 2 * nx * 20, bytesB = P.nblocks * nsw * 16 + 2 * nx * 16;
  if (tid == 0) {
    ccg_bar_init(barA, nsw);
    ccg_bar_init(barB, nsw);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sc.fail = 0;
  }
  __syncthreads();
  if (tid == 0) {
    ccg_bar_expect(barA, bytesA);
    ccg_bar_expect(barB, bytesB);
  }
  unsigned parity = 0;
  cg::this_cluster().sync();  // every block has started: its shared memory may be written
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
  double rr = ccg_sum(v, part, P, [](double t) { return t; });
  const double rr0 = rr, stop = ccg_stop(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  int status = -1, iter = 0, refA = fx_total_ref(rr0), refB = refA;
  if (isnan(rr)) status = TG_E_NAN;
  else if (!(rr >= stop) || rr == 0.0) status = TG_OK;
  auto tests = [&](double rn) { return cg_verdict(rn, stop, limit, iter + 1 >= a.maxiter); };
  if (tid == 0) sc.rr = rr;
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
    } else {
      inv_rr = 1.0 / rr;
    }
    __syncthreads();
    double va = 0;
    if (site) {
      for (int i = tid; i < n; i += T) {
        int xp, xm;
        offsets(i, xp, xm);
        const double2 o = ccg_op64<0, MU0>(a.km, pf, wt, wx, nx + i, nx, xp, xm);
        const FxC f = to_fx(o);
        ccg_store_send(qm, P, nx, i, make_longlong2(f.re, f.im), barA);
        ccg_store_send(qe, P, nx, i, f.e, barA);
        va = fma(o.x, o.x, va);
        va = fma(o.y, o.y, va);
      }
      ccg_post(va, refA, postA, P, nsw, barA);
    }
    ccg_bar_wait(barA, parity, &sc.fail);
    auto apply = [&](int i) {
      int xp, xm;
      offsets(i, xp, xm);
      return ccg_op64<1, MU0>(a.kd, qf, wt, wx, nx + i, nx, xp, xm);
    };
    double2 ap = make_double2(0.0, 0.0);  // the thread's first site, before alpha is known
    if (site) {
      if (tid < n) ap = apply(tid);
    } else {
      double pap;
      const bool ok = fx_partials_total(postA, P.nblocks * nsw, refA, pap);
      if (tid == T) {
        sc.alpha = div_newton(rr, pap);
        sc.okA = ok;
        sc.refA = fx_total_ref(pap);
        ccg_bar_expect(barA, bytesA);  // of the next iteration
      }
    }
    __syncthreads();
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    double alpha = sc.alpha;
    refA = sc.refA;
    if (!sc.okA) {
      const double pap = ccg_sum(va, part, P, [](double t) { return t; });
      alpha = sc.rr / pap;
      refA = fx_total_ref(pap);
    }
    double vb = 0;
    if (site) {
      for (int i = tid; i < n; i += T) {
        if (i != tid) ap = apply(i);
        double2 xv = x[i], rv = r[nx + i];
        const double2 pv = p[nx + i];
        rv.x -= alpha * ap.x;
        rv.y -= alpha * ap.y;
        ccg_store_send(r, P, nx, i, rv, barB);
        vb = fma(rv.x, rv.x, vb);
        vb = fma(rv.y, rv.y, vb);
        xv.x += alpha * pv.x;
        xv.y += alpha * pv.y;
        x[i] = xv;
      }
      ccg_post(vb, refB, postB, P, nsw, barB);
    }
    ccg_bar_wait(barB, parity, &sc.fail);
    if (!site) {
      double rn;
      const bool ok = fx_partials_total(postB, P.nblocks * nsw, refB, rn);
      if (tid == T) {
        sc.beta = div_prepared(rn, rr, inv_rr);
        sc.verdict = tests(rn);
        sc.okB = ok;
        sc.refB = fx_total_ref(rn);
        sc.rn = rn;
        ccg_bar_expect(barB, bytesB);
      }
    }
    __syncthreads();
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    parity ^= 1u;
    beta = sc.beta;
    status = sc.verdict;
    refB = sc.refB;
    if (!sc.okB) {
      const double rn = ccg_sum(vb, part, P, [](double t) { return t; });
      beta = rn / sc.rr;
      status = tests(rn);
      refB = fx_total_ref(rn);
      __syncthreads();
      if (tid == 0) sc.rn = rn;
      __syncthreads();
    }
    iter += 1;
    if (!site) {  // the last reads of sc.rr and sc.rn before this are behind a block barrier
      rr = sc.rn;
      if (tid == T) sc.rr = rr;
    }
  }
  ccg_leave(status == TG_E_TIMEOUT);
  for (int i = tid; i < n; i += blockDim.x) a.x[P.b0 + i] = x[i];
  ccg_report(a.st, a.log, a.log_index, iter > 0 ? sc.rn : rr, rr0, stop, iter, 0, status);
}

// Mixed: the iteration and the FP64 reliable update of k_pcgmx.  The FP64 x, its
// image M x and the FP64 links stay in global memory (a reliable update is one
// in about fifty iterations); reads of what other blocks wrote there go to L2.
template <bool MU0> __global__ void __launch_bounds__(kCcgThreads + 32, 1) k_ccgmx(PcgMxArgs a, int wmax, int nmax) {
  extern __shared__ __align__(16) unsigned char ccg_smem[];
  __shared__ CcgScalars sc;
  __shared__ __align__(8) unsigned long long bars[2];
  const Geo& g = a.g;
  const CcgPart P = ccg_part(g.V);
  const int nx = g.nx, n = P.n, win = n + 2 * nx, T = blockDim.x - 32, tid = threadIdx.x, nsw = T >> 5;
  const bool site = tid < T;  // else: the scalar warp
  longlong2* postA = reinterpret_cast<longlong2*>(ccg_smem);
  longlong2* postB = postA + kCcgPart;
  double* part = reinterpret_cast<double*>(postB + kCcgPart);
  float2* p = reinterpret_cast<float2*>(part + kCcgPart);
  float2* q = p + wmax;
  float2* r = q + wmax;
  float2* wt = r + wmax;
  float2* wx = wt + wmax;
  float2* xs = wx + wmax;

  const unsigned barA = ccg_smem_addr(&bars[0]), barB = ccg_smem_addr(&bars[1]);
  const unsigned bytesA = P.nblocks * nsw * 16 + 2 * nx * 8, bytesB = P.nblocks * nsw * 16 + 2 * nx * 8;
  if (tid == 0) {
    ccg_bar_init(barA, nsw);
    ccg_bar_init(barB, nsw);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sc.fail = 0;
  }
  __syncthreads();
  if (tid == 0) {
    ccg_bar_expect(barA, bytesA);
    ccg_bar_expect(barB, bytesB);
  }
  unsigned parity = 0;
  cg::this_cluster().sync();  // every block has started: its shared memory may be written
  double v = 0;
  for (int j = tid; j < win; j += blockDim.x) {
    int s = P.b0 - nx + j;
    s += (s < 0) ? g.V : (s >= g.V ? -g.V : 0);
    const double2 bb = a.b[s];
    const float2 rb = make_float2((float)bb.x, (float)bb.y);
    r[j] = rb;
    p[j] = rb;
    wt[j] = a.Wt32[s];
    wx[j] = a.Wx32[s];
    if (j >= nx && j < nx + n) {
      xs[j - nx] = make_float2(0.f, 0.f);
      v = fma(bb.x, bb.x, v);
      v = fma(bb.y, bb.y, v);
    }
  }
  for (int i = tid; i < n; i += blockDim.x) a.x[P.b0 + i] = make_double2(0.0, 0.0);
  double rr = ccg_sum(v, part, P, [](double t) { return t; });
  const double rr0 = rr, stop = ccg_stop(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  double drop = kRuDrop * rr;  // |r|^2 below which a reliable update is due
  int status = -1, iter = 0, n_ru = 0, since_ru = 0, refA = fx_total_ref(rr0), refB = refA;
  if (isnan(rr)) status = TG_E_NAN;
  else if (!(rr >= stop) || rr == 0.0) status = TG_OK;
  auto due = [&](double rn) -> int {  // a reliable update
    return since_ru + 1 >= a.ru_interval || iter + 1 >= a.maxiter || cg_update_due(rn, stop, drop, limit);
  };
  if (tid == 0) sc.rr = rr;
  int xp0, xm0;  // of the thread's first site
  ccg_x_offsets(g, min(P.b0 + tid, g.V - 1), xp0, xm0);
  auto offsets = [&](int i, int& xp, int& xm) {
    xp = xp0;
    xm = xm0;
    if (i != tid) ccg_x_offsets(g, P.b0 + i, xp, xm);
  };
  float bf = 0.f;
  while (status < 0) {
    double inv_rr = 0;
    if (site) {
      for (int j = tid; j < win; j += T) {
        const float2 rv = r[j], pv = p[j];
        p[j] = make_float2(fmaf(bf, pv.x, rv.x), fmaf(bf, pv.y, rv.y));
      }
    } else {
      inv_rr = 1.0 / rr;
    }
    __syncthreads();
    float va = 0;
    if (site) {
      for (int i = tid; i < n; i += T) {
        int xp, xm;
        offsets(i, xp, xm);
        const float2 o = ccg_op32<0, MU0>(a.km32, p, wt, wx, nx + i, nx, xp, xm);
        va = fmaf(o.x, o.x, va);
        va = fmaf(o.y, o.y, va);
        ccg_store_send(q, P, nx, i, o, barA);
      }
      ccg_post(va, refA, postA, P, nsw, barA);
    }
    ccg_bar_wait(barA, parity, &sc.fail);
    auto apply = [&](int i) {
      int xp, xm;
      offsets(i, xp, xm);
      return ccg_op32<1, MU0>(a.kd32, q, wt, wx, nx + i, nx, xp, xm);
    };
    float2 ap = make_float2(0.f, 0.f);  // the thread's first site, before alpha is known
    if (site) {
      if (tid < n) ap = apply(tid);
    } else {
      double pap;
      const bool ok = fx_partials_total(postA, P.nblocks * nsw, refA, pap);
      if (tid == T) {
        sc.af = (float)div_newton<false>(rr, pap);
        sc.okA = ok;
        sc.refA = fx_total_ref(pap);
        ccg_bar_expect(barA, bytesA);  // of the next iteration
      }
    }
    __syncthreads();
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    float af = sc.af;
    refA = sc.refA;
    if (!sc.okA) {
      const double pap = ccg_sum((double)va, part, P, [](double t) { return t; });
      af = (float)(sc.rr / pap);
      refA = fx_total_ref(pap);
    }
    float vb = 0;
    if (site) {
      for (int i = tid; i < n; i += T) {
        if (i != tid) ap = apply(i);
        float2 xv = xs[i], rv = r[nx + i];
        const float2 pv = p[nx + i];
        rv.x = fmaf(-af, ap.x, rv.x);
        rv.y = fmaf(-af, ap.y, rv.y);
        ccg_store_send(r, P, nx, i, rv, barB);
        vb = fmaf(rv.x, rv.x, vb);
        vb = fmaf(rv.y, rv.y, vb);
        xv.x = fmaf(af, pv.x, xv.x);
        xv.y = fmaf(af, pv.y, xv.y);
        xs[i] = xv;
      }
      ccg_post(vb, refB, postB, P, nsw, barB);
    }
    ccg_bar_wait(barB, parity, &sc.fail);
    if (!site) {
      double rn;
      const bool ok = fx_partials_total(postB, P.nblocks * nsw, refB, rn);
      if (tid == T) {
        sc.bf = (float)(rn * inv_rr);
        sc.verdict = due(rn);
        sc.okB = ok;
        sc.refB = fx_total_ref(rn);
        sc.rn = rn;
        ccg_bar_expect(barB, bytesB);
      }
    }
    __syncthreads();
    if (sc.fail) {
      status = TG_E_TIMEOUT;
      break;
    }
    parity ^= 1u;
    bf = sc.bf;
    refB = sc.refB;
    int need = sc.verdict;
    if (!sc.okB) {
      const double rn = ccg_sum((double)vb, part, P, [](double t) { return t; });
      bf = (float)(rn / sc.rr);
      need = due(rn);
      refB = fx_total_ref(rn);
      __syncthreads();
      if (tid == 0) sc.rn = rn;
      __syncthreads();
    }
    iter += 1;
    since_ru += 1;
    if (!need) {
      if (!site) {  // the last reads of sc.rr and sc.rn before this are behind a block barrier
        rr = sc.rn;
        if (tid == T) sc.rr = rr;
      }
      continue;
    }
    rr = sc.rn;
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
    cg::this_cluster().sync();
    auto ld_x = [&](int s) { return __ldcg(a.x + s); };
    if (site)
      for (int i = tid; i < n; i += T) {
        int t, x;
        double2 own;
        site_tx(g, P.b0 + i, t, x);
        a.tmp[P.b0 + i] = dslash_ld<double, 0, MU0>(g, a.km, ld_x, a.Wt, a.Wx, P.b0 + i, t, x, own);
      }
    cg::this_cluster().sync();
    double vt = 0;
    auto ld_t = [&](int s) { return __ldcg(a.tmp + s); };
    if (site)
      for (int i = tid; i < n; i += T) {
        int t, x;
        double2 own;
        const int s = P.b0 + i;
        site_tx(g, s, t, x);
        const double2 ap64 = dslash_ld<double, 1, MU0>(g, a.kd, ld_t, a.Wt, a.Wx, s, t, x, own), bb = a.b[s];
        const double2 rv = make_double2(bb.x - ap64.x, bb.y - ap64.y);
        ccg_store(r, P, nx, i, make_float2((float)rv.x, (float)rv.y));
        vt = fma(rv.x, rv.x, vt);
        vt = fma(rv.y, rv.y, vt);
      }
    const double rt = ccg_sum(vt, part, P, [](double t) { return t; });
    if (rt > kRuRestart * rr) bf = 0.f;  // the recursive residual was far too optimistic: restart p from r
    drop = kRuDrop * rt;
    rr = rt;
    if (tid == 0) sc.rr = sc.rn = rt;  // read again after the next block barrier
    since_ru = 0;
    n_ru += 1;
    if (isnan(rt)) status = TG_E_NAN;
    else if (rt < stop) status = TG_OK;
    else if (rt > limit) status = TG_E_DIVERGED;
    else if (iter >= a.maxiter) status = TG_E_NOCONV;
  }
  ccg_leave(status == TG_E_TIMEOUT);
  ccg_report(a.st, a.log, a.log_index, rr, rr0, stop, iter, n_ru, status);
}

// ---------------------------------------------------------------------------
// Launch
// ---------------------------------------------------------------------------
// shared memory of a block: the sums' partials, the window, the own sites
static size_t ccg_bytes(const Geo& g, int nblocks, bool mixed) {
  const size_t nmax = (g.V + nblocks - 1) / nblocks, win = nmax + 2 * (size_t)g.nx;
  return kCcgPart * (2 * sizeof(longlong2) + sizeof(double)) + win * (mixed ? kCcg32Window : kCcg64Window) +
         nmax * (mixed ? kCcg32Own : kCcg64Own);
}

// the largest cluster of these kernels that the current device can run (16 is
// not a portable size), 0 if it cannot tell
static int ccg_max_cluster() {
  static std::mutex mu;
  static std::unordered_map<int, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(dev);
  if (it != cache.end()) return it->second;
  int best = 0;
  const void* kernels[] = {(const void*)k_ccg64<true>, (const void*)k_ccg64<false>, (const void*)k_ccgmx<true>,
                           (const void*)k_ccgmx<false>};
  bool ok = true;
  for (const void* k : kernels)
    ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCcgSmem) == cudaSuccess &&
         cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  for (int c = kCcgMaxBlocks; ok && best == 0 && c >= 1; c /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(kCcgThreads + 32);
    cfg.dynamicSmemBytes = kCcgSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    best = c;
    for (const void* k : kernels) {
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 1) best = 0;
    }
  }
  (void)cudaGetLastError();  // a size that is refused is not an error of the caller's
  cache.emplace(dev, best);
  return best;
}

// The cluster's shape for a lattice, or none.  About 64 sites a block, up to 16
// blocks: a pass is bound by its own latency until then (us per FP64 / mixed
// iteration at 1, 2, 4, 8, 16 blocks: 16^2 4.0 / 2.6, 3.3 / 2.5, 3.3 / 2.4, 3.3 / 2.5,
// 3.3 / 2.6; at 4, 8, 16: 32^2 4.0 / 2.5, 3.2 / 2.3, 3.0 / 2.3; 64^2 9.5 / 3.8,
// 6.2 / 3.5, 4.3 / 2.9), a block owns at least a row.  One site per thread in
// FP64, two to four in the mixed solver beyond 256 sites a block, whose shorter
// passes gain less from more warps than the sums lose (96^2 at 512 / 256
// threads: FP64 7.8 / 7.7, mixed 4.0 / 3.5).  It gives way to the grid's
// shared memory at 512 sites a block in FP64 and 2400 mixed (gcg_shape, with the figures of
// both); its own limits, 850 and 3300, are where the solver of tg_pcg.cu was met
// (128^2 FP64 9.8 / 9.3, 256^2 mixed 7.6 / 7.1), and hold where the grid's is turned off.
// TG_CLUSTER_CG=0 turns it off, =blocks:threads sets the shape; the overrides of
// the grid solvers (TG_PCG_BLOCK, TG_MIXED_CG) turn it off as well.
CcgShape ccg_shape(const Geo& g, bool mixed) {
  const CcgShape none{0, 0};
  if (getenv("TG_PCG_BLOCK") != nullptr || getenv("TG_MIXED_CG") != nullptr) return none;
  const char* e = getenv("TG_CLUSTER_CG");
  int want = 1, threads = 0;
  while (want < kCcgMaxBlocks && want * 128 <= g.V) want *= 2;
  if (e && sscanf(e, "%d:%d", &want, &threads) >= 1 && want <= 0) return none;
  // (the lattice's limits first: a large one never asks the device)
  const int blocks = std::min(std::min(want, kCcgMaxBlocks), g.nt), n = (g.V + blocks - 1) / blocks;
  if (ccg_bytes(g, blocks, mixed) > (size_t)kCcgSmem || n > (mixed ? 3300 : 850)) return none;
  if (blocks > ccg_max_cluster()) return none;
  const int own = mixed && n > 256 ? std::max(256, n / 4) : n;
  const int t = threads > 0 ? threads : own;
  return CcgShape{blocks, std::min(kCcgThreads, (t + 31) / 32 * 32)};
}

template <class K, class Args> static cudaError_t ccg_launch(K kernel, cudaStream_t s, const Args& a, bool mixed,
                                                             const CcgShape& sh) {
  const int nmax = (a.g.V + sh.blocks - 1) / sh.blocks;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sh.blocks);
  cfg.blockDim = dim3((unsigned)sh.threads + 32);  // and the scalar warp
  cfg.dynamicSmemBytes = ccg_bytes(a.g, sh.blocks, mixed);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)sh.blocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, a, nmax + 2 * a.g.nx, nmax);
}

cudaError_t ccg64(cudaStream_t s, bool mu0, const Pcg64Args& a, const CcgShape& sh) {
  return mu0 ? ccg_launch(k_ccg64<true>, s, a, false, sh) : ccg_launch(k_ccg64<false>, s, a, false, sh);
}
cudaError_t ccgmx(cudaStream_t s, bool mu0, const PcgMxArgs& a, const CcgShape& sh) {
  return mu0 ? ccg_launch(k_ccgmx<true>, s, a, true, sh) : ccg_launch(k_ccgmx<false>, s, a, true, sh);
}

}  // namespace tg
