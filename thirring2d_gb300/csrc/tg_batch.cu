// tg_batch.cu -- the batched-chain kernel's instances with one thread block
// per chain, the instance table the autotuner chooses from, and dispatch
// (cluster instances: tg_batch_cluster.cu).
#include <algorithm>

#include "tg_batch_impl.cuh"

namespace tg {

template <int BS, int MINB, BatchSolves S>
__global__ void __launch_bounds__(BS, MINB) k_batch_trajectory(const BatchChain* __restrict__ chains,
                                                               const int* __restrict__ order, int n,
                                                               BatchFields F, BatchTraj P, ChainResult* results,
                                                               unsigned long long* queue) {
  batch_trajectory_body<BlockTeam, S>(chains, order, n, F, P, results, queue);
}

// The kernel instances the autotuner chooses from: (threads per block,
// minimum resident blocks per SM).  More blocks per SM cap the registers (64 at
// 2048 resident threads, with spills in the column march); fewer leave room
// for the march's registers (up to 255 at 256 threads and one block).
// The cluster instances split each chain over 2 or 4 SMs; their variants with
// solo_sites hand the chains of up to 64^2 or 96^2 sites (the end of the
// largest-first queue) to single blocks, which no longer wait on cluster
// barriers.
const BatchCfg kBatchCfgs[kBatchNumCfgs] = {
    {128, 8, 1, 0},    {256, 4, 1, 0},    {256, 2, 1, 0},    {256, 1, 1, 0},    {384, 1, 1, 0},
    {512, 1, 1, 0},    {512, 1, 2, 0},    {512, 1, 4, 0},    {256, 1, 4, 0},    {512, 1, 2, 4096},
    {512, 1, 2, 9216}, {512, 1, 4, 4096}, {512, 1, 4, 9216}, {256, 1, 4, 4096}, {256, 1, 4, 9216},
    {512, 1, 4, 4096, 1}};

// the cluster kernel of instance cfg (see batch_cluster_max)
static int cluster_kernel_of(int cfg) {
  const BatchCfg& c = kBatchCfgs[cfg];
  if (c.pairs) return 3;
  return c.cluster == 2 ? 0 : (c.block == 512 ? 1 : 2);
}

template <int BS, int MINB, BatchSolves S = kSolvesBoth> const void* batch_kernel() {
  return (const void*)k_batch_trajectory<BS, MINB, S>;
}

// The kernel that runs instance cfg.  The 64-register ones (8 blocks of 128 or 4 of
// 256 threads per SM) run FP64 trajectories at 128 registers and half the
// blocks: the integer limbs of the FP64 operator need about 125 in the march and
// spill 2 KB at 64.  64 chains of 16^2 ... 128^2 at 4 blocks of 256:
// 296 ms so, 549 at 64 registers; 512 chains of 16^2 at 8 blocks of 128: 5.3, 7.6.
static const void* batch_kernel_of(int cfg, bool fp64) {
  switch (cfg) {
    case 0: return fp64 ? batch_kernel<128, 4, kSolvesFp64>() : batch_kernel<128, 8, kSolvesMixed>();
    case 1: return fp64 ? batch_kernel<256, 2>() : batch_kernel<256, 4, kSolvesMixed>();
    case 2: return batch_kernel<256, 2>();
    case 3: return batch_kernel<256, 1>();
    case 4: return batch_kernel<384, 1>();
    default: return batch_kernel<512, 1>();
  }
}
static int batch_min_blocks(int cfg, bool fp64) {
  return fp64 && cfg <= 1 ? kBatchCfgs[cfg].minb / 2 : kBatchCfgs[cfg].minb;
}

// One block's share of an SM's shared memory at its minimum resident blocks, less
// the kernels' static part and the 1 KB the hardware keeps per block.
int batch_smem_limit(int cfg) {
  const int per_block = 228 * 1024 / (kBatchCfgs[cfg].cluster > 1 ? 1 : batch_min_blocks(cfg, true));
  return std::min(per_block - 1024, 227 * 1024) - kBatchStaticSmem;
}

// Let kernel k of instance cfg have up to the instance's share.  The limit belongs to
// the kernel, not to a launch: one that followed the launch's own need would be lowered by
// another batch's thread between the two.  (All instances that run one kernel have
// the same share.)
void batch_allow_smem(const void* k, int cfg) {
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, batch_smem_limit(cfg));
}

static void launch_kernel(cudaStream_t s, const void* k, int cfg, int grid, int block, const BatchChain* chains,
                          const int* order, int n, const BatchFields& F, const BatchTraj& P, ChainResult* results,
                          unsigned long long* queue) {
  const int sm = P.cg.smem;
  if (sm > 0) batch_allow_smem(k, cfg);
  BatchFields f = F;
  BatchTraj p = P;
  void* args[] = {&chains, &order, &n, &f, &p, &results, &queue};
  cudaLaunchKernel(k, dim3((unsigned)grid), dim3((unsigned)block), args, (size_t)sm, s);
}

int batch_teams(int cfg, int sms, bool fp64) {
  if (kBatchCfgs[cfg].cluster > 1) return batch_cluster_max(cluster_kernel_of(cfg));
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batch_kernel_of(cfg, fp64), kBatchCfgs[cfg].block, 0) !=
      cudaSuccess)
    return 0;
  return nb * sms;
}

int batch_filler_blocks(int cfg, int sms) {
  const BatchCfg& c = kBatchCfgs[cfg];
  if (c.cluster <= 1 || c.solo_sites <= 0) return 0;
  const int clusters = batch_cluster_max(cluster_kernel_of(cfg));
  return std::max(0, sms - clusters * c.cluster);
}

void batch_filler_launch(cudaStream_t s, int cfg, int blocks, const BatchChain* chains, const int* order, int n,
                         const BatchFields& F, const BatchTraj& P, ChainResult* results, unsigned long long* queue) {
  BatchTraj f = P;
  f.from_back = 1;
  // the one-block instance of the cluster kernel's block size: its solo chains
  // run the same code, so a chain's result does not depend on which block ran it
  const int bs = kBatchCfgs[cfg].block;
  launch_kernel(s, bs == 512 ? batch_kernel<512, 1>() : batch_kernel<256, 1>(), cfg, blocks, bs, chains, order, n, F, f, results,
                queue);
}

void batch_trajectory(cudaStream_t s, int cfg, int sms, const BatchChain* chains, const int* order, int n,
                      const BatchFields& F, const BatchTraj& P, ChainResult* results, unsigned long long* queue) {
  const int teams = std::min(n, std::max(1, batch_teams(cfg, sms, P.cg.precision == TG_PREC_FP64)));
  if (kBatchCfgs[cfg].cluster > 1)
    batch_cluster_launch(s, cfg, cluster_kernel_of(cfg), teams, chains, order, n, F, P, results, queue);
  else
    launch_kernel(s, batch_kernel_of(cfg, P.cg.precision == TG_PREC_FP64), cfg, teams, kBatchCfgs[cfg].block, chains, order, n, F,
                  P, results, queue);
}

}  // namespace tg
