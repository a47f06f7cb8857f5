"""The integer sums of one-block chains (block_sum_int in csrc/tg_batch_impl.cuh) by
themselves: a sum whose scale does not fit is taken again in FP64, and the next
one goes by the new scale, in every thread."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <vector>
#include "tg_batch_impl.cuh"
using namespace tg;
// total k is made of 1 / blockDim.x of it in every thread; out[k] the sum, refs[k][thread] the scale after it
__global__ void k_sums(const double* totals, int n, int ref0, double* out, int* refs) {
  int ref = ref0;
  for (int k = 0; k < n; k++) {
    const double t = block_sum_int(totals[k] / blockDim.x, ref, [](double s) { return s; });
    if (threadIdx.x == 0) out[k] = t;
    refs[k * blockDim.x + threadIdx.x] = ref;
  }
}
int main() {  // threads, sums, first scale's total; totals -> sums, scales, expected scales
  double h[3];
  if (fread(h, sizeof h, 1, stdin) != 1) return 1;
  const int threads = (int)h[0], n = (int)h[1];
  std::vector<double> v(n), out(n);
  std::vector<int> refs(n * threads);
  if (fread(v.data(), 8, n, stdin) != (size_t)n) return 1;
  double *dv, *dout;
  int* dr;
  if (cudaMalloc(&dv, 8 * n) || cudaMalloc(&dout, 8 * n) || cudaMalloc(&dr, 4 * n * threads)) return 2;
  cudaMemcpy(dv, v.data(), 8 * n, cudaMemcpyHostToDevice);
  k_sums<<<1, threads>>>(dv, n, fx_total_ref(h[2]), dout, dr);
  if (cudaMemcpy(out.data(), dout, 8 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  cudaMemcpy(refs.data(), dr, 4 * n * threads, cudaMemcpyDeviceToHost);
  for (int k = 0; k < n; k++) {
    int lo = refs[k * threads], hi = lo;
    for (int t = 0; t < threads; t++) {
      lo = refs[k * threads + t] < lo ? refs[k * threads + t] : lo;
      hi = refs[k * threads + t] > hi ? refs[k * threads + t] : hi;
    }
    const double r[4] = {out[k], (double)lo, (double)hi, (double)fx_total_ref(out[k])};
    fwrite(r, sizeof r, 1, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("bsum")
    (d / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(d / "h"), str(d / "h.cu")],
                   check=True, capture_output=True)
    return str(d / "h")


@pytest.mark.parametrize("threads", [32, 128, 256, 512])
@pytest.mark.parametrize("totals", [[1.0, 0.9, 1e-3, 1.1e-3, 0.7e-3, 5e-4],     # a drop past the scale, then on
                                    [1.0, 1e9, 0.8e9, 3.0, 2.5, 2.0],           # growth past it, and a drop
                                    [1.0, 0.0, 2.0, 1.5, np.nan, 2.0, 1.0],     # totals that give no scale
                                    [1.0, 1e-300, 1.0, 1.0]])
def test_sums_go_on_after_a_refused_one(harness, threads, totals):
    """The sum to 2^-50 (integer terms: threads * 2^-62; FP64: under 16 roundings), and the
    scale of that sum in all threads."""
    v = np.array(totals)
    out = np.frombuffer(subprocess.run([harness], input=np.array([threads, len(v), 1.0]).tobytes() + v.tobytes(),
                                       capture_output=True, check=True).stdout).reshape(-1, 4)
    assert np.allclose(out[:, 0], v, rtol=2.0 ** -49, atol=0, equal_nan=True)
    assert np.array_equal(out[:, 1], out[:, 3]) and np.array_equal(out[:, 2], out[:, 3])
