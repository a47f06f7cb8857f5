// tg_onchip.cuh -- what the CG solvers that keep a lattice in shared memory have in
// common (tg_cluster_cg.cu: one cluster; tg_grid_cg.cu: the whole grid): a block's share
// of the sites with a window of its neighbours, the operator on it, and the scalars
// that a warp without sites hands to the others.
#pragma once

#include "tg_device.cuh"
#include "tg_scalar.cuh"

namespace tg {

constexpr int kCcgThreads = 512;               // most site threads of a block (one more warp does the scalars)
constexpr int kCcgSmem = 224 * 1024;           // dynamic shared memory a block may use

// The block's share of the lattice.
struct CcgPart {
  int nblocks, c, b0, n;  // own sites b0 .. b0 + n - 1
  int prev, next, nprev;  // the neighbouring blocks, the previous one's site count
};
__device__ __forceinline__ CcgPart ccg_part(int V) {
  CcgPart p;
  p.nblocks = (int)gridDim.x;
  p.c = (int)blockIdx.x;
  auto at = [&](int c) { return (int)((long long)V * c / p.nblocks); };
  p.b0 = at(p.c);
  p.n = at(p.c + 1) - p.b0;
  p.prev = p.c == 0 ? p.nblocks - 1 : p.c - 1;
  p.next = p.c == p.nblocks - 1 ? 0 : p.c + 1;
  p.nprev = at(p.prev + 1) - at(p.prev);
  return p;
}

template <typename T> __device__ __forceinline__ T ccg_warp_allsum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void ccg_report(CgState* st, CgLog* log, int log_index, double rr, double rr0, double stop,
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

__device__ __forceinline__ double ccg_stop(double rr0, double rel_tol, double abs_tol2) {
  double stop = abs_tol2;
  if (rel_tol > 0 && rel_tol * rel_tol * rr0 > stop) stop = rel_tol * rel_tol * rr0;
  return stop;
}

// Offsets from a site to its x neighbours in the t-major order.
__device__ __forceinline__ void ccg_x_offsets(const Geo& g, int s, int& xp, int& xm) {
  int t, x;
  site_tx(g, s, t, x);
  xp = (x == g.nx - 1) ? 1 - g.nx : 1;
  xm = (x == 0) ? g.nx - 1 : -1;
}

// Block-floating operands (tg_fixed.cuh) in shared memory.
struct FxArr {
  longlong2* m;
  int* e;
  __device__ __forceinline__ FxC get(int i) const {
    const longlong2 v = m[i];
    return FxC{v.x, v.y, e[i]};
  }
};

template <int DAG, bool MU0>
__device__ __forceinline__ double2 ccg_op64(const OpK<double>& k, const FxArr& v, const FxLink* wt, const FxLink* wx,
                                            int j, int nx, int xp, int xm) {
  const FxC c = v.get(j), tu = v.get(j + nx), td = v.get(j - nx), xu = v.get(j + xp), xd = v.get(j + xm);
  const FxLink a = wt[j], b = wt[j - nx], p = wx[j], q = wx[j + xm];
  double2 o;
  if (!fx_dslash<DAG, MU0>(k, c, tu, td, xu, xd, a, b, p, q, o)) {
    // (a vector that is zero in places has many such sites; fx_value takes denormals for zeros)
    if ((c.e | tu.e | td.e | xu.e | xd.e) == 0 && fx_finite(k, a, b, p, q)) return make_double2(0.0, 0.0);
    o = dslash_vals<double, DAG, MU0>(k, fx_value(c), fx_value(tu), fx_value(td), fx_value(xu), fx_value(xd),
                                      fx_link_value(a), fx_link_value(b), fx_link_value(p), fx_link_value(q));
  }
  return o;
}

// bytes of shared memory per window site and per own site
constexpr int kCcg64Window = 6 * 16 + 2 * 4, kCcg64Own = 16;
constexpr int kCcg32Window = 5 * 8, kCcg32Own = 8;

template <int DAG, bool MU0>
__device__ __forceinline__ float2 ccg_op32(const OpK<float>& k, const float2* v, const float2* wt, const float2* wx,
                                           int j, int nx, int xp, int xm) {
  return dslash_vals<float, DAG, MU0>(k, v[j], v[j + nx], v[j - nx], v[j + xp], v[j + xm], wt[j], wt[j - nx], wx[j],
                                      wx[j + xm]);
}

// What the scalar warp hands to the block after the sums: the first sum's step
// length, the second's beta and verdict (FP64: a status or -1 to go on; mixed:
// whether a reliable update is due), and the scales of the next sums.
struct CcgScalars {
  double alpha, beta;
  float af, bf;
  int okA, refA, okB, refB, verdict, fail;
  double rr, rn;  // |r|^2 before and after the iteration, for a sum that is taken again
};

}  // namespace tg
