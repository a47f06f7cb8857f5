"""The partials of the launch-per-iteration reductions (grid_sum): every kernel that
reduces stores one per block, and the blocks it may be launched with must not
exceed what tg_create allocates -- on the CPU, over marching widths with strips
from nine tenths full, the widths and heights around them, and one site per
thread; and the solver that launches the most blocks, on the GPU, at such a width."""
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "thirring2d_gb300", "csrc")

HARNESS = r"""
#include <cstdio>
#include "tg_internal.cuh"
using namespace tg;
int main() {  // records nt, nx, march allowed -> march, blocks of partials
  int r[3];
  while (fread(r, sizeof r, 1, stdin) == 1) {
    Geo g{};
    g.nt = r[0]; g.nx = r[1]; g.V = r[0] * r[1];
    g.march = r[2] && march_ok(g.nx);
    const int out[2] = {g.march, reduction_blocks(g)};
    fwrite(out, sizeof out, 1, stdout);
  }
}
"""


def test_partials_cover_every_launch(tmp_path):
    (tmp_path / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{CSRC}", f"-I{ROOT}/include", "-o", str(tmp_path / "h"), str(tmp_path / "h.cu")], check=True,
                   capture_output=True)
    nxs = list(range(2, 400)) + [448, 512, 516, 518, 550, 1000, 1024, 1375, 2000, 2048]
    rec = np.array([(nt, nx, m) for nx in nxs for nt in (2, 3, 8, 64, 517, 519, 720, 1377, 4000) for m in (0, 1)
                    if nt * nx < 1 << 24], np.int32)
    out = np.frombuffer(subprocess.run([str(tmp_path / "h")], input=rec.tobytes(), capture_output=True, check=True).stdout,
                        np.int32).reshape(-1, 2)
    ragged = 0
    for (nt, nx, _), (march, blocks) in zip(rec.tolist(), out.tolist()):
        sites = -(-nt * nx // 256)
        rows = -(-(-(-nx // 32) * nt) // 8) if march else 0   # warp rows of 32 columns, eight warps a block
        ragged += rows > sites + 32
        assert blocks >= max(sites, rows), (nt, nx)
    assert ragged > 50   # more blocks than sites / 256 with a margin: what the workspace was once sized for
    assert re.search(r"red\.partials, \(size_t\)reduction_blocks\(L->g\)\)", open(os.path.join(CSRC, "tg_capi.cu")).read())


@pytest.mark.gpu
@pytest.mark.parametrize("nt,nx", [(720, 144), (517, 144), (519, 176), (1377, 58), (64, 29)])
@pytest.mark.parametrize("precision", [0, 1])
def test_launch_solver_at_ragged_widths(nt, nx, precision):
    """Launched and persistent solves of one system to 1e-11: they differ by 4e-11 / m at most."""
    import thirring2d_gb300 as tg
    rng = np.random.default_rng(nx)
    A, m = rng.normal(0, 0.4, (nt, nx, 2)), 0.3
    b = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
    with tg.Lattice(nt, nx, m, 0.5, 0.1, -1, -1) as L:
        L.set_gauge(A)
        got = [L.fmdm_invert_cg(b, tg.cg_params(rel_tol=1e-11, abs_tol2=0, precision=precision, solver=s))
               for s in (tg.native.SOLVER_LAUNCHES, tg.native.SOLVER_PERSISTENT)]
        eta = L.stochastic_md_action(b)
        assert np.isfinite(eta)
    assert got[0][1].status == got[1][1].status == 0
    assert np.linalg.norm(got[0][0] - got[1][0]) <= 4e-11 / m * np.linalg.norm(got[1][0])
