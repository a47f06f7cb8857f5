"""The prefetched FP64 march (march_ring64 in csrc/tg_stencil.cuh), audited on the CPU with its own
index functions, strips that are not full among them: every address that a lane fetches lies
inside the lattice and is the one its step needs, and a slot is not fetched into before
the step that reads it is over."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "tg_stencil.cuh"
using namespace tg;
constexpr int D = kMarchT, EL = 2 * kMarchT;
#define CHECK(c) do { if (!(c)) { printf("nt %d nx %d strip %d rows %d-%d lane %d: %s\n", nt, nx, xw, ta, tb, lane, #c); exit(1); } } while (0)
static long long audit(int nt, int nx, int xw, int ta, int tb, int lane) {
  const Strip p = strip_of(nx, xw, lane);
  const int n = tb - ta, V = nt * nx, want = xw * 32 + lane;
  CHECK(p.x0 == xw * 32 && p.last >= 0 && p.last < 32 && p.x0 + p.last < nx);
  CHECK(lane > p.last || p.x == want);
  CHECK(p.xle == (p.x0 + nx - 1) % nx && p.xre == (p.x0 + p.last + 1) % nx);
  int row[D], edge[2][2], groups = 0, edge_group[2], row_group[D];   // what each slot holds, and since which group
  auto issue = [&](int i) {
    const int t = ta + i, slot = ring_slot(i), so = t * nx + p.x, sp = row_above(nt, t) * nx + p.x;
    CHECK(so >= 0 && so < V && sp >= 0 && sp < V && sp == ((t + 1) % nt) * nx + p.x);
    row[slot] = i;
    row_group[slot] = groups;
    if (i % kMarchT == 0 && lane < EL) {
      const int c = ring_edge(nx, p, t, tb, lane), es = ring_edge_slot(i);
      CHECK(c >= 0 && c < V);
      edge[es][0] = i / kMarchT;
      edge[es][1] = c;
      edge_group[es] = groups;
    }
  };
  for (int i = 0; i < D - 1; i++) {
    if (i < n) issue(i);
    groups++;
  }
  for (int i = 0; i < n; i++) {   // the march's steps: fetch ahead, wait for all groups but the last D - 1, read
    if (i + D - 1 < n) issue(i + D - 1);
    groups++;
    const int done = groups - (D - 1);
    CHECK(row[ring_slot(i)] == i && row_group[ring_slot(i)] < done);
    if (lane < EL) {
      const int chunk = i / kMarchT, es = ring_edge_slot(i);
      // (read with the chunk's first row; the lane's own row of the chunk, as far as the range goes)
      if (i % kMarchT == 0) CHECK(edge[es][0] == chunk && edge_group[es] < done);
      const int t = ta + chunk * kMarchT + lane % kMarchT;
      if (i % kMarchT == 0 && t < tb) CHECK(edge[es][1] == t * nx + (lane < kMarchT ? p.xle : p.xre));
    }
  }
  return n;
}
int main() {
  const int nxs[] = {29, 30, 31, 32, 58, 63, 64, 95, 96, 300, 322, 1000}, nts[] = {2, 3, 4, 5, 7, 8, 13, 40};
  long long steps = 0;
  for (int nx : nxs)
    for (int nt : nts) {
      if (!march_ok(nx)) { printf("%d does not march\n", nx); return 1; }
      for (int xw = 0; xw < march_strips(nx); xw++)
        for (int ta = 0; ta < nt; ta++)
          for (int tb = ta + 1; tb <= nt; tb += (tb - ta < 6 ? 1 : 5))
            for (int lane = 0; lane < 32; lane++) steps += audit(nt, nx, xw, ta, tb, lane);
    }
  printf("ok %lld\n", steps);
}
"""


def test_every_fetch_and_slot(tmp_path):
    (tmp_path / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(tmp_path / "h"), str(tmp_path / "h.cu")],
                   check=True, capture_output=True)
    out = subprocess.run([str(tmp_path / "h")], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout


@pytest.mark.parametrize("name", ["strip_of(nx, xw, lane)", "row_above(g.nt, t)", "ring_edge(nx, st, t, tb, lane)", "ring_edge_slot(i0)"])
def test_the_march_uses_them(name):
    src = open(os.path.join(ROOT, "thirring2d_gb300", "csrc", "tg_stencil.cuh")).read()
    assert name in src[src.index("march_ring64("):]
