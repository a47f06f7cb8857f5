"""How a CG iteration ends (cg_verdict in csrc/tg_scalar.cuh): on the CPU against the
plain comparisons, NaNs of either sign and payload among them; and on the GPU,
solves that meet a NaN inside the iteration in every solver."""
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OK, NOCONV, DIVERGED, NAN = 0, 1, 2, 3

HARNESS = r"""
#include <cstdio>
#include "tg_scalar.cuh"
int main() {  // records rn, stop, limit, last -> verdict, update due (drop = stop / 2)
  double r[4];
  while (fread(r, sizeof r, 1, stdin) == 1) {
    const int out[2] = {tg::cg_verdict(r[0], r[1], r[2], r[3] != 0), tg::cg_update_due(r[0], r[1], r[1] / 2, r[2])};
    fwrite(out, sizeof out, 1, stdout);
  }
}
"""


def test_verdicts(tmp_path):
    (tmp_path / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(tmp_path / "h"), str(tmp_path / "h.cu")],
                   check=True, capture_output=True)
    nans = np.array([0x7FF8000000000000, 0xFFF8000000000000, 0x7FFFFFFFFFFFFFFF, 0xFFFFFFFFFFFFFFFF, 0x7FF0000000000001,
                     0xFFF0000000000001], np.uint64).view(np.float64)
    values = np.concatenate((nans, [0.0, -0.0, 5e-324, 1e-310, 1e-30, 1.0, 2.0, 1e10, 1e300, np.inf]))
    bounds = [0.0, 5e-324, 1e-30, 1.0, 1e10, np.inf]
    rec = np.array([(0, s, lim, last) for _ in values for s in bounds for lim in bounds for last in (0.0, 1.0)])
    rec[:, 0] = np.repeat(values, len(bounds) ** 2 * 2)
    out = np.frombuffer(subprocess.run([str(tmp_path / "h")], input=rec.tobytes(), capture_output=True, check=True).stdout,
                        np.int32).reshape(-1, 2)
    for (rn, stop, limit, last), (v, due) in zip(rec, out):
        want = NAN if np.isnan(rn) else OK if rn < stop else DIVERGED if rn > limit else NOCONV if last else -1
        assert v == want
        assert bool(due) == bool(np.isnan(rn) or rn < stop or rn > limit)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nt,nx", [(8, 8), (48, 64), (128, 128), (256, 256), (512, 640)])
def test_nan_inside_a_solve(nt, nx, precision):
    """M b = 0 exactly (m = 0, A = 0, periodic sides, a constant b): |M p|^2 = 0, alpha is
    infinite and r - alpha 0 NaN; and a b whose |b|^2 overflows."""
    import thirring2d_gb300 as tg
    cp = tg.cg_params(rel_tol=1e-10, abs_tol2=0, precision=precision)
    with tg.Lattice(nt, nx, 0.0, 0.5, 0.0, 1, 1) as L:
        for value in (1.0, 0.37 + 0.21j):
            b = np.full((nt, nx), value, complex)
            assert not L.fm_mul(b).any()
            assert L.fmdm_invert_cg(b, cp)[1].status == tg.native.TG_E_NAN
    rng = np.random.default_rng(3)
    with tg.Lattice(nt, nx, 0.3, 0.5, 0.0, -1, 1) as L:
        L.set_gauge(rng.normal(0, 0.5, (nt, nx, 2)))
        b = 1e160 * (rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx)))
        assert L.fmdm_invert_cg(b, cp)[1].status == tg.native.TG_E_NAN


QUOTIENTS = r"""
#include <cstdio>
#include "tg_scalar.cuh"
int main() {  // records a, b -> a / b with 1 / b known
  double r[2];
  while (fread(r, sizeof r, 1, stdin) == 1) {
    const double q = tg::div_prepared(r[0], r[1], 1.0 / r[1]);
    fwrite(&q, sizeof q, 1, stdout);
  }
}
"""


def test_quotients_from_a_reciprocal(tmp_path):
    """(1/2 + 2^-40) ulp, 0.75 allowed, as of the other quotients; down to sums that are denormal,
    whose reciprocal overflows."""
    (tmp_path / "h.cu").write_text(QUOTIENTS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(tmp_path / "h"), str(tmp_path / "h.cu")],
                   check=True, capture_output=True)
    rng = np.random.default_rng(2)
    e = rng.integers(-1074, 900, 4000)
    e[:200] = rng.integers(-1074, -1000, 200)
    b = rng.uniform(1, 2, 4000) * np.exp2(e.astype(float))
    b = b[b > 0]
    a = b * rng.uniform(1e-3, 4, len(b))
    got = np.frombuffer(subprocess.run([str(tmp_path / "h")], input=np.stack([a, b], 1).tobytes(), capture_output=True,
                                       check=True).stdout)
    for x, y, v in zip(a, b, got):
        q = Fraction(x) / Fraction(y)
        assert abs(Fraction(float(v)) - q) <= Fraction(3, 4) * Fraction(math.ulp(float(v)))


@pytest.mark.gpu
@pytest.mark.parametrize("nt,nx", [(8, 8), (48, 64), (128, 128), (256, 256), (512, 640)])
def test_tiny_sources(nt, nx):
    """|b|^2 of 1e-295 to 1e-300 and a residual whose square ends below the normal range."""
    import thirring2d_gb300 as tg
    rng = np.random.default_rng(3)
    with tg.Lattice(nt, nx, 0.3, 0.5, 0.0, -1, 1) as L:
        L.set_gauge(rng.normal(0, 0.5, (nt, nx, 2)))
        b = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
        cp = tg.cg_params(rel_tol=1e-8, abs_tol2=0, maxiter=2000)
        x, res = L.fmdm_invert_cg(b, cp)
        y, tiny = L.fmdm_invert_cg(1e-150 * b, cp)
    assert res.status == tiny.status == 0
    assert abs(tiny.iterations - res.iterations) <= 2
    assert np.linalg.norm(y / 1e-150 - x) <= 4e-8 / 0.3 * np.linalg.norm(x)
