// tg_pcg.cu -- the persistent CG solver: one cooperative launch runs a whole
// solve of M^dag M x = b (fmdm_invert_cg, hmc.c:341-404), FP64 or FP32 with
// FP64 reliable updates, instead of two launches per iteration.
//
// All blocks are co-resident (cooperative launch) and meet at a grid barrier
// after each reduction.  Every block writes its partial sum, passes the
// barrier, and then adds all partials in a fixed order itself, so every block
// holds the same bitwise total and takes the same branch: control flow stays
// uniform across the grid without a broadcast.  Two partial arrays alternate,
// so a block that races ahead never overwrites partials another block is
// still reading.  Vectors that other blocks write during the solve are read
// with ld.global.cg (L2), so no SM sees a stale L1 line (a one-block grid reads
// them through L1, see ldv).  Each block marches
// the same row ranges in every phase (tg_stencil.cuh).
//
// The barrier's wait is bounded: after kBarrierSpinLimit polls a block gives
// up, the solve ends with TG_E_TIMEOUT, and every other block times out at
// its next barrier, so a fault in the scheme cannot hang the GPU.
#include <math.h>
#include <stdlib.h>

#include <algorithm>

#include "tg_fused.cuh"
#include "tg_gridbar.cuh"
#include "tg_resident.h"
#include "tg_scalar.cuh"

namespace tg {

// Threads per block of the persistent kernels (512 / BS blocks per SM, 128
// registers): one block of 512 threads per SM on lattices that fill the GPU --
// fewer arrivals at each grid barrier -- and two of 256 on smaller ones, whose
// rows would otherwise occupy too few SMs (pcg_launch).
constexpr int pcg_min_blocks(int bs) { return 512 / bs; }

__device__ __forceinline__ bool grid_barrier_n(const GridBar& b, unsigned nblocks, long long limit) {
  __shared__ int s_ok;
  if (nblocks == 1) {
    __syncthreads();
    return true;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const bool ok = warp0_grid_wait(b, nblocks, limit);
    if (threadIdx.x == 0) s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ bool grid_barrier(const GridBar& b) {
  return grid_barrier_n(b, gridDim.x, kBarrierSpinLimit);
}

// The barrier's failure path, for tests: one barrier that also waits for
// `phantom` blocks that do not exist gives up after `limit` polls; status[0]
// = TG_OK if it was passed, TG_E_TIMEOUT if it gave up.
__global__ void k_barrier_check(GridBar b, unsigned phantom, long long limit, int* status) {
  if (threadIdx.x == 0) barrier_epoch() = 0;
  const bool ok = grid_barrier_n(b, gridDim.x + phantom, limit);
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = ok ? TG_OK : TG_E_TIMEOUT;
}

// Loads of vectors that the solve itself writes.  Across blocks they go to L2
// (ld.global.cg), so no SM reads a stale L1 line; in a one-block grid (ONE)
// the block barriers order every write before every later read, and the loads
// may hit L1: a 16^2 lattice's vectors (a few tens of KB) then stay on chip.
template <bool ONE, typename T> __device__ __forceinline__ T ldv(const T* p) {
  if constexpr (ONE) return *p;
  else return __ldcg(p);
}

// Warp 0's read of the blocks' partials after a grid barrier: NP values per
// block, part[NP * i + k].  Each lane adds the blocks lane, lane + 32, ... in
// index order, with the loads of up to 256 blocks issued before any is used,
// then a fixed shuffle tree; the totals are valid in lane 0.  Measured 0.17 us
// faster per sum than a read by all threads with a block-wide tree.
template <int NP>
__device__ __forceinline__ void warp_read_partials(const double* part, double (&tot)[NP]) {
  const int lane = threadIdx.x & 31, nb = (int)gridDim.x;
#pragma unroll
  for (int k = 0; k < NP; k++) tot[k] = 0.0;
  for (int j0 = 0; j0 < nb; j0 += 256) {
    double v[8][NP];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int i = j0 + lane + 32 * j;
#pragma unroll
      for (int k = 0; k < NP; k++) v[j][k] = (i < nb) ? __ldcg(part + NP * i + k) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int k = 0; k < NP; k++) tot[k] += v[j][k];
  }
#pragma unroll
  for (int k = 0; k < NP; k++) tot[k] = warp_sum(tot[k]);
}

// Grid total of the threads' partials v (added in their own precision within
// a block, as the launch path's kernels do, and in FP64 across blocks, in the
// fixed order of warp_read_partials), handed to f, which runs in thread 0 of
// every block; every thread of the block gets f's result.  The scalars that
// follow a sum (alpha, beta, the stopping tests) are thus computed once per
// block: a double division is about ten operations of the FP64 pipe, which
// retires two per SM per clock.
// Two block barriers in all: one after the warps' sums (it also orders the
// block's writes before the arrival), one to hand the result to the block.
template <int BS, typename T, class F, class Prep = NoPrep>
__device__ __forceinline__ bool grid_total_then(T v, double* part, const GridBar& bar, F f, decltype(f(0.0))& out,
                                                Prep prep = {}) {
  using S = decltype(f(0.0));
  __shared__ T sh[BS / 32];
  __shared__ S s_out;
  __shared__ int s_ok;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    T b = (lane < BS / 32) ? sh[lane] : T(0);
    b = warp_sum(b);
    if (gridDim.x == 1) {  // a one-block grid: its total is the grid's, no round trip through memory
      if (lane == 0) {
        prep();
        s_out = f((double)b);
        s_ok = 1;
      }
    } else {
      if (lane == 0) part[blockIdx.x] = (double)b;
      const bool ok = warp0_grid_wait(bar, gridDim.x, kBarrierSpinLimit, prep);
      if (ok) {
        double s[1];
        warp_read_partials<1>(part, s);
        if (lane == 0) s_out = f(s[0]);
      }
      if (lane == 0) s_ok = ok;
    }
  }
  __syncthreads();
  out = s_out;
  return s_ok != 0;
}

// ---------------------------------------------------------------------------
// Fixed-point grid sums (the mixed CG's two iteration sums, FP32 partials).
// The barrier and the data travel in one 64-bit word per kind of sum: each
// block adds, with one release-add, its arrival (bits 0-8), an overflow flag
// (bits 9-17) and its block total as an integer at the scale 2^e (bits 18-63),
// then polls the word with acquire loads until the arrivals since its previous
// use of the word (the difference to the value it read then) number the grid.
// Integer addition is associative, so every block reads the same total in
// any order of arrival: the result stays deterministic.  That saves the read
// of the partials after the barrier, one L2 round trip (measured 1.1 us of
// 2.8 per sum with 152 blocks).
//
// The scale (a power of two) follows the last total of the same kind: block totals near 2^29,
// so a block total may grow 256-fold (to 2^37; 511 blocks at most, the sum
// field holds 46 bits) before it overflows.  A block whose total would
// overflow (or is not finite) sets its flag instead; a grid total below
// 2^26 per block would carry a rounding error (half a unit per block) above
// 2^-27 of itself, about the error of an FP32 block total.  In either case
// every block takes the exact path: it adds the FP32 block totals, which each
// block also writes to `part`, in FP64 (warp_read_partials).  Consecutive uses
// of one word are separated by a sum of the other kind, which no block passes
// before every block has read the word, so no block reads the other use's
// additions.  The words are 0 at launch.
// ---------------------------------------------------------------------------
// 2^e for |e| <= 1000, from its bits (no FP64 arithmetic)
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

struct FxSum {
  unsigned long long* word;
  unsigned long long last;  // the word's value at this block's previous read
  double scale, inv;        // block totals are added as rint(total * scale); inv = 1 / scale
  // The scale for the next sum from a total of the same kind: 2^(29 -
  // log2(total / grid)), from the exponent bits (all blocks compute the same
  // scale from the same total; FP64 arithmetic is slow on this GPU).
  __device__ __forceinline__ void rescale(double total) {
    if (!(total > 0.0) || !isfinite(total)) return;
    const int lt = ((__double2hiint(total) >> 20) & 0x7ff) - 1023;
    const int lg = 31 - __clz((int)gridDim.x);
    const int e = min(max(29 - (lt - lg), -1000), 1000);
    scale = pow2(e);
    inv = pow2(-e);
  }
};
constexpr int kFxOvfShift = 9, kFxSumShift = 18;
constexpr unsigned kFxMaxGrid = 511;
constexpr double kFxBlockCap = 137438953472.0;  // 2^37
constexpr int kFxMinBits = 26;                   // the exact path below 2^26 per block

template <int BS, class F, class Prep = NoPrep>
__device__ __forceinline__ bool grid_total_fx(float v, double* part, const GridBar& bar, FxSum& fx, F f,
                                              decltype(f(0.0))& out, Prep prep = {}) {
  using S = decltype(f(0.0));
  if (gridDim.x == 1 || gridDim.x > kFxMaxGrid) return grid_total_then<BS>(v, part, bar, f, out, prep);
  __shared__ float sh[BS / 32];
  __shared__ S s_out;
  __shared__ int s_ok;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sh[wid] = v;
  __syncthreads();  // the warps' sums, and the block's writes before the arrival
  if (wid == 0) {
    float b = (lane < BS / 32) ? sh[lane] : 0.f;
    b = warp_sum(b);
    const unsigned nb = gridDim.x;
    int ok = 1, exact = 0;
    double total = 0;
    if (lane == 0) {
      part[blockIdx.x] = (double)b;  // for the exact path
      const double sc = (double)b * fx.scale;
      const bool fits = sc >= 0.0 && sc < kFxBlockCap;  // false for NaN too
      const unsigned long long add =
          (fits ? ((unsigned long long)__double2ll_rn(sc) << kFxSumShift) : (1ull << kFxOvfShift)) | 1ull;
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(fx.word), "l"(add) : "memory");
      prep();
      unsigned long long cur, d;
      long long spins = 0;
      while (true) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(cur) : "l"(fx.word) : "memory");
        d = cur - fx.last;
        if ((unsigned)(d & kFxMaxGrid) == nb) break;
        if (++spins > kBarrierSpinLimit) {
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
      fx.last = cur;
      const unsigned long long fsum = d >> kFxSumShift;
      exact = ((d >> kFxOvfShift) & kFxMaxGrid) != 0 || fsum < ((unsigned long long)nb << kFxMinBits);
      total = __ull2double_rn(fsum) * fx.inv;
    }
    __syncwarp();
    ok = __shfl_sync(0xffffffffu, ok, 0);
    exact = __shfl_sync(0xffffffffu, exact, 0);
    if (ok && exact) {
      double s[1];
      warp_read_partials<1>(part, s);
      total = s[0];
    }
    if (lane == 0) {
      if (ok) {
        fx.rescale(total);
        s_out = f(total);
      }
      s_ok = ok;
    }
  }
  __syncthreads();
  out = s_out;
  return s_ok != 0;
}

template <int BS>
__device__ __forceinline__ bool grid_total(double v, double* part, const GridBar& bar, double& out) {
  return grid_total_then<BS>(v, part, bar, [](double t) { return t; }, out);
}

// What the iterations need after their sums.
struct PcgTail64 {
  double rn, beta;
  int status;  // -1: go on
};
struct PcgTailMx {
  double rn;
  float bf;
  int need;  // a reliable update is due
};

__device__ __forceinline__ void pcg_report(CgState* st, CgLog* log, int log_index, double rr, double rr0, double stop,
                                           int iter, int n_ru, int status) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  st->rr = rr;
  st->rr0 = rr0;
  st->rr_true = rr;
  st->stop = stop;
  st->iter = iter;
  st->n_ru = n_ru;
  st->status = status;
  st->done = 1;
  st->need_ru = 0;
  st->restart = 0;
  st->log_index = log_index;
  if (log != nullptr && log_index >= 0) {
    CgLog& l = log[log_index];
    l.iter = iter;
    l.status = status;
    l.n_ru = n_ru;
    l.rr = rr;
    l.rr0 = rr0;
  }
}

__device__ __forceinline__ double stop_of(double rr0, double rel_tol, double abs_tol2) {
  double stop = abs_tol2;
  if (rel_tol > 0 && rel_tol * rel_tol * rr0 > stop) stop = rel_tol * rel_tol * rr0;
  return stop;
}

// ---------------------------------------------------------------------------
// FP64: the iteration of k_cg1 + k_cg2_64
// ---------------------------------------------------------------------------
// Rows in flight per warp in the FP64 march, and the shared memory they take
// (12.8 KB a warp, 205 KB a 512-thread block).  The prefetched march against one
// with two rows' loads in registers, us per iteration: 1024^2 53.2 / 58.7, 512^2
// 21.2 / 21.2.  16 warps per SM beat 12 (61.5 at 1024^2), 18 and 20 (62.5, 58.5: 88 B of
// spills); two rows per step, interleaved, gave 56.4.  A lattice that does not march is
// launched with the ring too: the L1 that it takes is no loss to one site per thread (2000x100
// 14.00 us with, 14.02 without; 3000x170 36.6, 36.8; 20000x40 52.3, 52.5).
constexpr int kRingRows = 4;
constexpr int kRingWarp = ring_bytes<kRingRows, 1, 3>() > ring_bytes<kRingRows, 2, 0>()
                              ? ring_bytes<kRingRows, 1, 3>() : ring_bytes<kRingRows, 2, 0>();
template <int BS, bool MU0, bool ONE = false>
__global__ void __launch_bounds__(BS, pcg_min_blocks(BS)) k_pcg64(Pcg64Args a) {
  extern __shared__ __align__(16) unsigned char pcg_ring[];
  unsigned char* const ring = pcg_ring + (threadIdx.x >> 5) * kRingWarp;
  if (threadIdx.x == 0) barrier_epoch() = 0;
  const Geo& g = a.g;
  double* partA = a.part;
  double* partB = a.part + gridDim.x;
  double v = 0;
  TG_SITES(s, g.V) {  // x = 0, r = p = b (hmc.c:352-357)
    const double2 bb = a.b[s];
    a.x[s] = make_double2(0.0, 0.0);
    a.r[s] = bb;
    a.p0[s] = bb;
    v = fma(bb.x, bb.x, v);
    v = fma(bb.y, bb.y, v);
  }
  double rr = 0;
  int status = -1, iter = 0;
  if (!grid_total<BS>(v, partB, a.bar, rr)) status = TG_E_TIMEOUT;
  const double rr0 = rr;
  const double stop = stop_of(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  if (status < 0) {
    if (isnan(rr)) status = TG_E_NAN;
    else if (!(rr >= stop) || rr == 0.0) status = TG_OK;  // hmc.c:359-361
  }
  double beta = 0;
  int half = 0;
  while (status < 0) {
    const double2* p_old = half ? a.p1 : a.p0;
    double2* p_new = half ? a.p0 : a.p1;
    double va = 0;
    auto ld_a = [&](int i) {
      const double2 rv = ldv<ONE>(a.r + i), pv = ldv<ONE>(p_old + i);
      return make_double2(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
    };
    auto epi_a = [&](int s, double2 o, double2 pc) {
      p_new[s] = pc;
      a.Mp[s] = o;
      va = fma(o.x, o.x, va);
      va = fma(o.y, o.y, va);
    };
    if (!ONE && g.march) {
      const double2* const src[2] = {a.r, p_old};
      auto comb = [&](const double2* v) { return make_double2(fma(beta, v[1].x, v[0].x), fma(beta, v[1].y, v[0].y)); };
      auto epi = [&](int s, double2 o, double2 pc, const double2*) { epi_a(s, o, pc); };
      for_warp_rows(g, [&](int xw, int ta, int tb) {
        march_ring64<0, MU0, kRingRows, 2, 0>(g, a.km, src, nullptr, comb, a.Wt, a.Wx, xw, ta, tb, epi, ring);
      });
    } else {
      stencil_ld<double, 0, MU0>(g, a.km, ld_a, a.Wt, a.Wx, epi_a);
    }
    double alpha;
    if (!grid_total_then<BS>(va, partA, a.bar, [&](double pap) { return div_newton(rr, pap); }, alpha)) {
      status = TG_E_TIMEOUT;
      break;
    }
    double vb = 0;
    auto ld_b = [&](int i) { return ldv<ONE>(a.Mp + i); };
    auto update = [&](int s, double2 ap, double2 xv, double2 pv, double2 rv) {
      xv.x += alpha * pv.x;
      xv.y += alpha * pv.y;
      rv.x -= alpha * ap.x;
      rv.y -= alpha * ap.y;
      a.x[s] = xv;
      a.r[s] = rv;
      vb = fma(rv.x, rv.x, vb);
      vb = fma(rv.y, rv.y, vb);
    };
    if (!ONE && g.march) {
      const double2* const src[1] = {a.Mp};
      const double2* const ext[3] = {a.x, p_new, a.r};
      auto comb = [](const double2* v) { return v[0]; };
      auto epi = [&](int s, double2 ap, double2, const double2* e) { update(s, ap, e[0], e[32], e[64]); };
      for_warp_rows(g, [&](int xw, int ta, int tb) {
        march_ring64<1, MU0, kRingRows, 1, 3>(g, a.kd, src, ext, comb, a.Wt, a.Wx, xw, ta, tb, epi, ring);
      });
    } else {
      auto epi = [&](int s, double2 ap, double2) {
        update(s, ap, ldv<ONE>(a.x + s), ldv<ONE>(p_new + s), ldv<ONE>(a.r + s));
      };
      stencil_ld<double, 1, MU0>(g, a.kd, ld_b, a.Wt, a.Wx, epi);
    }
    PcgTail64 e;
    double inv_rr = 0;  // thread 0's
    if (!grid_total_then<BS>(vb, partB, a.bar, [&](double rn) {
          PcgTail64 o{rn, div_prepared(rn, rr, inv_rr), -1};
          if (isnan(rn)) o.status = TG_E_NAN;
          else if (rn < stop) o.status = TG_OK;           // hmc.c:381
          else if (rn > limit) o.status = TG_E_DIVERGED;  // hmc.c:383-386
          else if (iter + 1 >= a.maxiter) o.status = TG_E_NOCONV;
          return o;
        }, e, [&]() { inv_rr = 1.0 / rr; })) {
      status = TG_E_TIMEOUT;
      break;
    }
    iter += 1;
    beta = e.beta;
    rr = e.rn;
    status = e.status;
    half ^= 1;
  }
  pcg_report(a.st, a.log, a.log_index, rr, rr0, stop, iter, 0, status);
}

// ---------------------------------------------------------------------------
// Mixed: the iteration of k_cg1<float> + k_cgmx2, and the reliable update of
// k_ru1..3 with the same triggers and restart rule.
// ---------------------------------------------------------------------------
template <int BS, bool MU0, bool ONE = false>
__global__ void __launch_bounds__(BS, pcg_min_blocks(BS)) k_pcgmx(PcgMxArgs a) {
  if (threadIdx.x == 0) barrier_epoch() = 0;
  const Geo& g = a.g;
  // consecutive sums never share an array: alpha A, beta B, reliable update C
  double* partA = a.part;
  double* partB = a.part + gridDim.x;
  double* partC = a.part + 2 * gridDim.x;
  double v = 0;
  TG_SITES(s, g.V) {
    const double2 bb = a.b[s];
    a.x[s] = make_double2(0.0, 0.0);
    const float2 rb = make_float2((float)bb.x, (float)bb.y);
    a.r[s] = rb;
    a.p0[s] = rb;
    a.xs[s] = make_float2(0.f, 0.f);
    v = fma(bb.x, bb.x, v);
    v = fma(bb.y, bb.y, v);
  }
  double rr = 0;
  int status = -1, iter = 0, n_ru = 0, since_ru = 0;
  if (!grid_total<BS>(v, partB, a.bar, rr)) status = TG_E_TIMEOUT;
  const double rr0 = rr;
  const double stop = stop_of(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  double rr_true = rr;
  if (status < 0) {
    if (isnan(rr)) status = TG_E_NAN;
    else if (!(rr >= stop) || rr == 0.0) status = TG_OK;
  }
  float bf = 0.f;
  int half = 0;
  // the iteration sums, fixed-point (grid_total_fx), one word per kind
  FxSum fxA{a.bar.fx, 0ull, 1.0, 1.0}, fxB{a.bar.fx + 1, 0ull, 1.0, 1.0};
  fxA.rescale(rr0);
  fxB.rescale(rr0);
  while (status < 0) {
    const float2* p_old = half ? a.p1 : a.p0;
    float2* p_new = half ? a.p0 : a.p1;
    float va = 0;
    auto ld_a = [&](int i) {
      const float2 rv = ldv<ONE>(a.r + i), pv = ldv<ONE>(p_old + i);
      return make_float2(fmaf(bf, pv.x, rv.x), fmaf(bf, pv.y, rv.y));
    };
    auto epi_a = [&](int s, float2 o, float2 pc) {
      p_new[s] = pc;
      a.Mp[s] = o;
      va = fmaf(o.x, o.x, va);
      va = fmaf(o.y, o.y, va);
    };
    stencil_ld<float, 0, MU0>(g, a.km32, ld_a, a.Wt32, a.Wx32, epi_a);
    float af;
    if (!grid_total_fx<BS>(va, partA, a.bar, fxA, [&](double pap) { return (float)div_newton<false>(rr, pap); }, af)) {
      status = TG_E_TIMEOUT;
      break;
    }
    float vb = 0;
    auto ld_b = [&](int i) { return ldv<ONE>(a.Mp + i); };
    auto epi_b = [&](int s, float2 ap, float2) {
      float2 xv = ldv<ONE>(a.xs + s), pv = ldv<ONE>(p_new + s), rv = ldv<ONE>(a.r + s);
      xv.x = fmaf(af, pv.x, xv.x);
      xv.y = fmaf(af, pv.y, xv.y);
      rv.x = fmaf(-af, ap.x, rv.x);
      rv.y = fmaf(-af, ap.y, rv.y);
      a.xs[s] = xv;
      a.r[s] = rv;
      vb = fmaf(rv.x, rv.x, vb);
      vb = fmaf(rv.y, rv.y, vb);
    };
    stencil_ld<float, 1, MU0>(g, a.kd32, ld_b, a.Wt32, a.Wx32, epi_b);
    PcgTailMx e;
    double inv_rr = 0;  // thread 0's
    if (!grid_total_fx<BS>(vb, partB, a.bar, fxB, [&](double rn) {
          PcgTailMx o{rn, (float)(rn * inv_rr), 0};
          o.need = since_ru + 1 >= a.ru_interval || rn < stop || rn < kRuDrop * rr_true || iter + 1 >= a.maxiter ||
                   rn > limit || isnan(rn);
          return o;
        }, e, [&]() { inv_rr = 1.0 / rr; })) {
      status = TG_E_TIMEOUT;
      break;
    }
    iter += 1;
    since_ru += 1;
    bf = e.bf;
    rr = e.rn;
    half ^= 1;
    if (!e.need) continue;
    // reliable update: x += xs, xs = 0; r = b - M^dag M x in FP64; rs = (float) r
    TG_SITES(s, g.V) {
      const float2 d = ldv<ONE>(a.xs + s);
      double2 xv = ldv<ONE>(a.x + s);
      xv.x += (double)d.x;
      xv.y += (double)d.y;
      a.x[s] = xv;
      a.xs[s] = make_float2(0.f, 0.f);
    }
    if (!grid_barrier(a.bar)) {
      status = TG_E_TIMEOUT;
      break;
    }
    auto ld_x = [&](int i) { return ldv<ONE>(a.x + i); };
    auto epi_x = [&](int s, double2 o, double2) { a.tmp[s] = o; };
    stencil_ld<double, 0, MU0>(g, a.km, ld_x, a.Wt, a.Wx, epi_x);
    if (!grid_barrier(a.bar)) {
      status = TG_E_TIMEOUT;
      break;
    }
    double vt = 0;
    auto ld_t = [&](int i) { return ldv<ONE>(a.tmp + i); };
    auto epi_t = [&](int s, double2 ap, double2) {
      const double2 bb = a.b[s];
      const double2 rv = make_double2(bb.x - ap.x, bb.y - ap.y);
      a.r[s] = make_float2((float)rv.x, (float)rv.y);
      vt = fma(rv.x, rv.x, vt);
      vt = fma(rv.y, rv.y, vt);
    };
    stencil_ld<double, 1, MU0>(g, a.kd, ld_t, a.Wt, a.Wx, epi_t);
    double rt;
    if (!grid_total<BS>(vt, partC, a.bar, rt)) {
      status = TG_E_TIMEOUT;
      break;
    }
    if (rt > kRuRestart * rr) bf = 0.f;  // the recursive residual was far too optimistic: restart p from r
    rr_true = rt;
    rr = rt;
    since_ru = 0;
    n_ru += 1;
    if (isnan(rt)) status = TG_E_NAN;
    else if (rt < stop) status = TG_OK;
    else if (rt / rr0 > 1e10) status = TG_E_DIVERGED;
    else if (iter >= a.maxiter) status = TG_E_NOCONV;
  }
  pcg_report(a.st, a.log, a.log_index, rr, rr0, stop, iter, n_ru, status);
}

// ---------------------------------------------------------------------------
// Mixed, single reduction: the same solve as k_pcgmx (FP32 iterations, FP64
// reliable updates with the same triggers and restart rule, the same stopping
// tests), with CG in the Chronopoulos-Gear form (A. T. Chronopoulos and
// C. W. Gear, J. Comput. Appl. Math. 25 (1989) 153): with A = M^dag M,
//   s_k = w_k + beta_k s_{k-1},  p_k = r_k + beta_k p_{k-1},
//   x_{k+1} = x_k + alpha_k p_k,  r_{k+1} = r_k - alpha_k s_k,  w_{k+1} = A r_{k+1},
//   gamma = (r_{k+1}, r_{k+1}),  delta = (r_{k+1}, A r_{k+1}) = |M r_{k+1}|^2,
//   beta_{k+1} = gamma / gamma_k,  alpha_{k+1} = gamma / (delta - beta_{k+1} gamma / alpha_k),
// so one grid sum (gamma and delta together) per iteration instead of two.
// An iteration runs in two phases:
//   A  the vector updates (s, p, x, r in place), site by site: no neighbours,
//      every load of a thread's sites issued before the first store;
//   B  after a grid barrier, w = A r in one pass of the fused M^dag M march
//      (tg_fused.cuh), which also forms the partials of gamma and delta.
// Column-march lattices only.
// ---------------------------------------------------------------------------
struct PlainOp {
  float2 v;
};
struct PlainLd {  // the fused march's operand: r itself
  using Op = PlainOp;
  const float2* r;
  __device__ __forceinline__ Op own(int i) const { return Op{__ldcg(r + i)}; }
  __device__ __forceinline__ float2 val(int i) const { return __ldcg(r + i); }
};

__device__ __forceinline__ float2 axpy2(float a, float2 x, float2 y) {
  return make_float2(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y));
}
__device__ __forceinline__ float4 axpy4(float a, float4 x, float4 y) {
  return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

// Phase A over two sites per float4, one float4 per thread and array in flight
// (U = 1: the kernel then needs no local memory at all; U = 2 spilled 32-48 B
// and was 0.9% slower per iteration at 2048^2, U = 3 spilled 112 B and was 7%
// slower).
__device__ __forceinline__ void cgcg_update(const Geo& g, float4* __restrict__ r, const float4* __restrict__ w,
                                            float4* __restrict__ s, float4* __restrict__ p, float4* __restrict__ xs,
                                            float al, float be) {
  constexpr int U = 1;
  const int n4 = g.V >> 1;
  const int stride = gridDim.x * blockDim.x;
  for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n4; i0 += U * stride) {
    float4 rv[U], wv[U], sv[U], pv[U], xv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * stride;
      if (i < n4) {
        rv[u] = __ldcg(r + i);
        wv[u] = __ldcg(w + i);
        sv[u] = __ldcg(s + i);
        pv[u] = __ldcg(p + i);
        xv[u] = __ldcg(xs + i);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * stride;
      if (i < n4) {
        const float4 sk = axpy4(be, sv[u], wv[u]);
        const float4 pk = axpy4(be, pv[u], rv[u]);
        s[i] = sk;
        p[i] = pk;
        xs[i] = axpy4(al, pk, xv[u]);
        r[i] = axpy4(-al, sk, rv[u]);
      }
    }
  }
  if ((g.V & 1) && blockIdx.x == 0 && threadIdx.x == 0) {  // the last site of an odd number
    const int i = g.V - 1;
    float2 *const r2 = reinterpret_cast<float2*>(r), *const s2 = reinterpret_cast<float2*>(s),
           *const p2 = reinterpret_cast<float2*>(p), *const x2 = reinterpret_cast<float2*>(xs);
    const float2 rv = __ldcg(r2 + i), sk = axpy2(be, __ldcg(s2 + i), __ldcg(reinterpret_cast<const float2*>(w) + i)),
                 pk = axpy2(be, __ldcg(p2 + i), rv);
    s2[i] = sk;
    p2[i] = pk;
    x2[i] = axpy2(al, pk, __ldcg(x2 + i));
    r2[i] = axpy2(-al, sk, rv);
  }
}

// Grid totals of a pair of partials (gamma, delta): block sums in FP32,
// written to part as FP64 pairs; after the grid barrier, warp 0 of every block
// adds all blocks' pairs (warp_read_partials) and hands f of the totals, computed
// in its lane 0, to the block through one block barrier, two block barriers in
// all.  (Every thread computing alpha and beta itself took four FP64 divisions
// per thread and iteration, which the SM's FP64 pipe runs one warp at a time.)
template <int BS, class F, class Prep = NoPrep>
__device__ __forceinline__ bool grid_total2(float va, float vb, double* part, const GridBar& bar, F f,
                                            decltype(f(0.0, 0.0))& out, Prep prep = {}) {
  using S = decltype(f(0.0, 0.0));
  __shared__ float sha[BS / 32], shb[BS / 32];
  __shared__ S s_out;
  __shared__ int s_ok;
  va = warp_sum(va);
  vb = warp_sum(vb);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sha[wid] = va;
    shb[wid] = vb;
  }
  __syncthreads();
  if (wid == 0) {
    float a = (lane < BS / 32) ? sha[lane] : 0.f, b = (lane < BS / 32) ? shb[lane] : 0.f;
    a = warp_sum(a);
    b = warp_sum(b);
    if (lane == 0) {
      part[2 * blockIdx.x] = (double)a;
      part[2 * blockIdx.x + 1] = (double)b;
    }
    const bool ok = warp0_grid_wait(bar, gridDim.x, kBarrierSpinLimit, prep);
    if (ok) {
      double t[2];
      warp_read_partials<2>(part, t);
      if (lane == 0) s_out = f(t[0], t[1]);
    }
    if (lane == 0) s_ok = ok;
  }
  __syncthreads();
  out = s_out;
  return s_ok != 0;
}
// The FP64 reliable update shared by the single-reduction kernels:
// x += xs, xs = 0; r = (float)(b - M^dag M x) with |b - M^dag M x|^2 summed
// into rt.  False if a grid barrier gave up.
template <int BS, bool MU0, class Part>
__device__ __forceinline__ bool cgcg_reliable(const PcgMxArgs& a, float2* r, Part& part, double& rt) {
  const Geo& g = a.g;
  TG_SITES(s, g.V) {
    const float2 d = __ldcg(a.xs + s);
    double2 xv = __ldcg(a.x + s);
    xv.x += (double)d.x;
    xv.y += (double)d.y;
    a.x[s] = xv;
    a.xs[s] = make_float2(0.f, 0.f);
  }
  if (!grid_barrier(a.bar)) return false;
  auto ld_x = [&](int i) { return __ldcg(a.x + i); };
  auto epi_x = [&](int s, double2 o, double2) { a.tmp[s] = o; };
  stencil_ld<double, 0, MU0>(g, a.km, ld_x, a.Wt, a.Wx, epi_x);
  if (!grid_barrier(a.bar)) return false;
  double vt = 0;
  auto ld_t = [&](int i) { return __ldcg(a.tmp + i); };
  auto epi_t = [&](int s, double2 ap, double2) {
    const double2 bb = a.b[s];
    const double2 rv = make_double2(bb.x - ap.x, bb.y - ap.y);
    r[s] = make_float2((float)rv.x, (float)rv.y);
    vt = fma(rv.x, rv.x, vt);
    vt = fma(rv.y, rv.y, vt);
  };
  stencil_ld<double, 1, MU0>(g, a.kd, ld_t, a.Wt, a.Wx, epi_t);
  return grid_total<BS>(vt, part(), a.bar, rt);
}

// x = 0, r_0 = b, p_{-1} = s_{-1} = 0 and |b|^2 (shared set-up)
template <int BS, class Part>
__device__ __forceinline__ bool cgcg_start(const PcgMxArgs& a, float2* r, float2* p, float2* sv, Part& part,
                                           double& rr) {
  double v = 0;
  TG_SITES(s, a.g.V) {
    const double2 bb = a.b[s];
    a.x[s] = make_double2(0.0, 0.0);
    a.xs[s] = make_float2(0.f, 0.f);
    r[s] = make_float2((float)bb.x, (float)bb.y);
    p[s] = make_float2(0.f, 0.f);
    sv[s] = make_float2(0.f, 0.f);
    v = fma(bb.x, bb.x, v);
    v = fma(bb.y, bb.y, v);
  }
  return grid_total<BS>(v, part(), a.bar, rr);
}

__device__ __forceinline__ int ru_status(double rt, double stop, double rr0, int iter, int maxiter) {
  if (isnan(rt)) return TG_E_NAN;
  if (rt < stop) return TG_OK;
  if (rt / rr0 > 1e10) return TG_E_DIVERGED;
  if (iter >= maxiter) return TG_E_NOCONV;
  return -1;
}

// An iteration's scalars: (r, r), alpha, beta, and whether a reliable update is due.
struct CgcgStep {
  double gam, alpha, beta;
  int need;
};

template <int BS, bool MU0>
__global__ void __launch_bounds__(BS, pcg_min_blocks(BS)) k_pcgcg(PcgMxArgs a) {
  if (threadIdx.x == 0) barrier_epoch() = 0;
  const Geo& g = a.g;
  // Partial sums: two arrays of 2 * grid doubles (pairs; a single sum uses the
  // first half), used strictly in turn: a block that runs ahead to the next sum
  // writes the other array, never one that a slower block is still reading.
  int nsum = 0;
  auto part = [&]() { return a.part + 2 * gridDim.x * ((nsum++) & 1); };
  float2 *const r = a.r, *const w = a.w0, *const sv = a.s0, *const p = a.p0;
  double rr = 0;
  int status = -1, iter = 0, n_ru = 0, since_ru = 0;
  if (!cgcg_start<BS>(a, r, p, sv, part, rr)) status = TG_E_TIMEOUT;
  const double rr0 = rr;
  const double stop = stop_of(rr0, a.rel_tol, a.abs_tol2), limit = 1e10 * rr0;
  double rr_true = rr;
  if (status < 0) {
    if (isnan(rr)) status = TG_E_NAN;
    else if (!(rr >= stop) || rr == 0.0) status = TG_OK;
  }
  // phase B: w = A r; f of the totals of (r, r) and (r, A r) into out
  auto apply_sum = [&](auto f, CgcgStep& out, auto prep) -> bool {
    float ga = 0.f, de = 0.f;
    const PlainLd ld{r};
    auto epi = [&](int s, float2 wv, float2 u, const PlainOp& o) {
      w[s] = wv;
      ga = fmaf(o.v.x, o.v.x, fmaf(o.v.y, o.v.y, ga));
      de = fmaf(u.x, u.x, fmaf(u.y, u.y, de));
    };
    stencil_mdagm<MU0>(g, a.km32, a.kd32, ld, a.Wt32, a.Wx32, epi);
    return grid_total2<BS>(ga, de, part(), a.bar, f, out, prep);
  };
  double gam = 0, alpha = 0, beta = 0;
  CgcgStep st;
  if (status < 0) {
    if (apply_sum([](double gn, double dn) { return CgcgStep{gn, gn / dn, 0.0, 0}; }, st, NoPrep{})) {
      gam = st.gam;
      alpha = st.alpha;
    } else {
      status = TG_E_TIMEOUT;
    }
  }
  while (status < 0) {
    cgcg_update(g, reinterpret_cast<float4*>(r), reinterpret_cast<const float4*>(w), reinterpret_cast<float4*>(sv),
                reinterpret_cast<float4*>(p), reinterpret_cast<float4*>(a.xs), (float)alpha, (float)beta);
    double inv_gam = 0, inv_alpha = 0;  // thread 0's
    if (!grid_barrier(a.bar) || !apply_sum([&](double gn, double dn) {
          const double be = gn * inv_gam;
          const int need = since_ru + 1 >= a.ru_interval || gn < stop || gn < kRuDrop * rr_true ||
                           iter + 1 >= a.maxiter || gn > limit || isnan(gn) || isnan(dn);
          return CgcgStep{gn, div_newton(gn, dn - be * gn * inv_alpha), be, need};
        }, st, [&]() {
          inv_gam = 1.0 / gam;
          inv_alpha = 1.0 / alpha;
        })) {
      status = TG_E_TIMEOUT;
      break;
    }
    const int need = st.need;
    iter += 1;
    since_ru += 1;
    const double alpha_prev = alpha, gam_prev = gam;
    beta = st.beta;
    alpha = st.alpha;
    gam = rr = st.gam;
    if (!need) continue;
    // reliable update, then w = A r for the replaced r
    double rt;
    if (!cgcg_reliable<BS, MU0>(a, r, part, rt)) {
      status = TG_E_TIMEOUT;
      break;
    }
    const bool restart = rt > kRuRestart * rr;  // the recursive residual was far too optimistic
    rr_true = rt;
    rr = rt;
    since_ru = 0;
    n_ru += 1;
    status = ru_status(rt, stop, rr0, iter, a.maxiter);
    if (status >= 0) break;
    if (!apply_sum([&](double gn, double dn) {
          if (restart) return CgcgStep{gn, gn / dn, 0.0, 0};  // p and s restart from r and w
          const double be = gn / gam_prev;
          return CgcgStep{gn, gn / (dn - be * gn / alpha_prev), be, 0};
        }, st, NoPrep{})) {
      status = TG_E_TIMEOUT;
      break;
    }
    beta = st.beta;
    alpha = st.alpha;
    gam = st.gam;
  }
  pcg_report(a.st, a.log, a.log_index, rr, rr0, stop, iter, n_ru, status);
}

// ---------------------------------------------------------------------------
// Launchers: grid = co-resident blocks, at most the
// stencil's work; cooperative launch so the barrier cannot wait on a block
// that is not running.
// ---------------------------------------------------------------------------
template <class K, class Args>
cudaError_t coop_launch(K kernel, int grid, int bs, cudaStream_t s, const Args& a, int smem = 0) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)bs);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// Blocks of bs threads the stencil can use with at least `rows` rows of 32
// columns per warp (column march) or one site per thread.
int pcg_work(const Geo& g, int bs, int rows) {
  return g.march ? (march_strips(g.nx) * ((g.nt + rows - 1) / rows) + bs / 32 - 1) / (bs / 32) : nblocks(g.V, bs);
}

int pcg_grid(const Geo& g, int resident, int bs) {
  int grid = std::min(resident, pcg_work(g, bs, 1));
  if (grid > kPcgMaxGrid) grid = kPcgMaxGrid;
  return grid > 0 ? grid : 1;
}

// From how many sites on the persistent solvers march.  One site per thread starts
// each pass with all its loads, a march with its first rows'; its fewer loads and
// operations win when threads have three sites and more.  us per iteration, march /
// site by site: FP64 256^2 13.2 / 11.9, 384^2 17.1 / 16.3, 448^2 19.4 / 20.2, 512^2
// 21.8 / 24.5, 1000^2 51.3 / 64.3, 2048^2 168 / 266; mixed 256^2 8.3 / 7.1, 512^2 10.4 / 10.4,
// 768^2 14.6 / 14.7, 1024^2 18.9 / 21.4, 1000^2 19.3 / 20.8.
constexpr int kPcgMarch64 = 200000, kPcgMarchMx = 550000;

// TG_PCG_BLOCK=512 runs any lattice on the launch shape of a lattice that
// fills the GPU (one 512-thread block per SM, warps beyond the lattice's rows
// idle), so small test lattices can hold that shape to the reference's
// outputs; TG_PCG_BLOCK=256 forces the small-lattice shape.  Unset: by size.
int pcg_block_override() {
  const char* e = getenv("TG_PCG_BLOCK");
  if (e == nullptr) return 0;
  const int v = atoi(e);
  return (v == 512 || v == 256) ? v : 0;
}

// The 512-thread kernel when its blocks fill every SM with a row per warp (or a
// site per thread), else the 256-thread one.  A marching lattice spreads to one row
// per warp: its passes are bound by each warp's own latency, and more blocks cost
// the grid sums little (us per iteration at four rows / one row per warp: FP64 128^2
// 17.3 / 11.1, 256^2 17.4 / 13.5; mixed 256^2 9.4 / 8.6; blocks of 128 and 64 threads
// lose up to 8 us from 256^2 on).  A lattice whose work fits
// one 256-thread block at one_rows rows per warp runs the one-block instance
// (k1; L1-cached loads, block totals kept on chip): FP32 sums gain more from
// that than from four blocks (32^2 4.7 against 6.9 us), FP64 less (12.2, 10.1).
template <class K512, class K256, class K1, class Args>
cudaError_t pcg_launch(const Geo& g, K512 k512, K256 k256, K1 k1, int one_rows, cudaStream_t s, const Args& a,
                       int warp_smem = 0) {
  const int r512 = resident_blocks((const void*)k512, 512, 16 * warp_smem);
  const int r256 = resident_blocks((const void*)k256, 256, 8 * warp_smem);
  if (r512 <= 0 || r256 <= 0) return cudaErrorLaunchOutOfResources;
  const int force = pcg_block_override();  // (keeps the march: small lattices on the large ones' path)
  if (force == 512) return coop_launch(k512, std::min(r512, kPcgMaxGrid), 512, s, a, 16 * warp_smem);
  if (force == 0 && pcg_work(g, 512, 1) >= r512) return coop_launch(k512, pcg_grid(g, r512, 512), 512, s, a, 16 * warp_smem);
  if (one_rows > 0 && pcg_work(g, 256, one_rows) == 1) return coop_launch(k1, 1, 256, s, a);
  return coop_launch(k256, pcg_grid(g, r256, 256), 256, s, a, 8 * warp_smem);
}

cudaError_t pcg64(cudaStream_t s, bool mu0, Pcg64Args a) {
  if (a.g.V < kPcgMarch64 && pcg_block_override() == 0) a.g.march = 0;
  if (mu0) return pcg_launch(a.g, k_pcg64<512, true>, k_pcg64<256, true>, k_pcg64<256, true, true>, 1, s, a, kRingWarp);
  return pcg_launch(a.g, k_pcg64<512, false>, k_pcg64<256, false>, k_pcg64<256, false, true>, 1, s, a, kRingWarp);
}

cudaError_t barrier_check(cudaStream_t s, unsigned* count, unsigned phantom, long long limit, int* status) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(4);
  cfg.blockDim = dim3(64);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_barrier_check, GridBar{count}, phantom, limit, status);
}

cudaError_t pcgmx(cudaStream_t s, bool mu0, PcgMxArgs a) {
  if (a.g.V < kPcgMarchMx && pcg_block_override() == 0) a.g.march = 0;
  if (mu0) return pcg_launch(a.g, k_pcgmx<512, true>, k_pcgmx<256, true>, k_pcgmx<256, true, true>, kMarchT, s, a);
  return pcg_launch(a.g, k_pcgmx<512, false>, k_pcgmx<256, false>, k_pcgmx<256, false, true>, kMarchT, s, a);
}

cudaError_t pcgcg(cudaStream_t s, bool mu0, PcgMxArgs a) {
  if (!a.g.march) return cudaErrorInvalidValue;
  if (mu0) return pcg_launch(a.g, k_pcgcg<512, true>, k_pcgcg<256, true>, k_pcgcg<256, true>, 0, s, a);
  return pcg_launch(a.g, k_pcgcg<512, false>, k_pcgcg<256, false>, k_pcgcg<256, false>, 0, s, a);
}

}  // namespace tg
