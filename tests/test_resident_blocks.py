"""The resident blocks of a persistent kernel (csrc/tg_resident.h), on the CPU against a
fake CUDA runtime of two devices with different SM counts: the limit on dynamic shared
memory is each device's own and has to be raised there before a launch, and a
refusal is not a block count."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include "tg_resident.h"
static int dev = 0, refuse = 0, limit[2] = {48 * 1024, 48 * 1024};
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { *v = d == 0 ? 152 : 100; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int v) {
  if (refuse) return cudaErrorInvalidValue;
  limit[dev] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int threads, size_t smem) {
  *n = (int)smem <= limit[dev] ? 1024 / threads : 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}
int main() {
  static int kernel, other;
  for (dev = 0; dev < 2; dev++)
    for (int rep = 0; rep < 2; rep++) {
      const int n = tg::resident_blocks(&kernel, 512, 200000);
      printf("%d %d\n", n, limit[dev]);
    }
  dev = 0;
  printf("%d\n", tg::resident_blocks(&kernel, 256, 0));
  refuse = 1;
  printf("%d\n", tg::resident_blocks(&other, 512, 300000));
  refuse = 0;
  printf("%d\n", tg::resident_blocks(&other, 512, 100000));
}
"""


def test_each_device_gets_its_own_limit_and_count(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-cudart", "none", f"-I{ROOT}/thirring2d_gb300/csrc", "-o",
                    str(tmp_path / "h"), str(tmp_path / "h.cpp")], check=True, capture_output=True)
    out = subprocess.run([str(tmp_path / "h")], capture_output=True, check=True, text=True).stdout.split("\n")
    assert out[:7] == ["304 200000"] * 2 + ["200 200000"] * 2 + ["608", "0", "304"]
    src = {f: open(os.path.join(ROOT, "thirring2d_gb300", "csrc", f)).read() for f in ("tg_pcg.cu", "tg_kernels.cu")}
    for text in src.values():   # the launchers ask here, and keep no limit of their own
        assert "resident_blocks(" in text and "MaxDynamicSharedMemorySize" not in text
