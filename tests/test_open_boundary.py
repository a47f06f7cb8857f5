"""Open boundaries (bc = 0): what lies behind a link that is zero does not touch the site's
result, however large it is -- the FP64 operator's integer form on the CPU, and
both stencil paths on the GPU against the oracle."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include "tg_trig.cuh"
using namespace tg;
int main() {  // records: which link is open, angle, operand behind it -> accepted, W read back, the other links' marks
  double r[3];
  while (fread(r, sizeof r, 1, stdin) == 1) {
    FxLink q[4];
    double2 w;
    for (int i = 0; i < 4; i++) fx_link_of(r[1], i == (int)r[0] ? 0 : 1, w, q[i]);
    FxC v[5];
    for (int i = 0; i < 5; i++) v[i] = to_fx(i == (int)r[0] + 1 ? double2{r[2], r[2]} : double2{1.0, -0.5});
    double2 o;
    const bool ok = fx_dslash<0, true>(make_opk(0.1, 1, -1, true), v[0], v[1], v[2], v[3], v[4], q[0], q[1], q[2], q[3], o);
    const double2 z = fx_link_value(q[(int)r[0]]);
    const double out[5] = {(double)ok, z.x, z.y, o.x, o.y};
    fwrite(out, sizeof out, 1, stdout);
  }
}
"""


def test_an_open_link_is_not_summed_at_the_scale_behind_it(tmp_path):
    (tmp_path / "h.cu").write_text(HARNESS)
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-O1", "-gencode", "arch=compute_103a,code=sm_103a",
                    f"-I{ROOT}/thirring2d_gb300/csrc", f"-I{ROOT}/include", "-o", str(tmp_path / "h"), str(tmp_path / "h.cu")],
                   check=True, capture_output=True)
    values = (1.0, 0.0, 1e-320, 1e20, -1e200)
    rec = np.array([(k, a, v) for k in range(4) for a in (0.0, 0.3, -2.0, 5e6, np.nan, np.inf) for v in values])
    out = np.frombuffer(subprocess.run([str(tmp_path / "h")], input=rec.tobytes(), capture_output=True, check=True).stdout)
    want = {}
    for (k, a, v), (ok, zx, zy, x, y) in zip(rec, out.reshape(-1, 5)):
        if np.isfinite(a):
            assert ok == 1 and zx == 0 and zy == 0
            assert want.setdefault((k, a), (x, y)) == (x, y)   # whatever lies behind the link
        else:
            assert ok == 0 and np.isnan(zx) and np.isnan(zy)
    rec = np.array([(k, 0.3, v) for k in range(4) for v in (np.inf, -np.inf, np.nan)])   # 0 times these is NaN: the FP64 form
    out = np.frombuffer(subprocess.run([str(tmp_path / "h")], input=rec.tobytes(), capture_output=True, check=True).stdout)
    assert not out.reshape(-1, 5)[:, 0].any()


@pytest.mark.gpu
@pytest.mark.parametrize("nt,nx", [(2, 2), (3, 5), (6, 10), (8, 32), (33, 64), (40, 300)])
@pytest.mark.parametrize("bc", [(0, 1), (-1, 0), (0, 0)])
@pytest.mark.parametrize("mu", [0.0, 0.2])
def test_large_values_behind_an_open_boundary(oracle_lib, nt, nx, bc, mu):
    """The first row and column are 1e18 times the rest.  The integer form's 5 and the
    oracle's 18 roundings of at most 5 scales (50 of 2^-53), of the largest operand that a
    link connects to the site."""
    import thirring2d_gb300 as tg
    rng = np.random.default_rng(nt * 1000 + nx)
    A, m = rng.normal(0, 0.7, (nt, nx, 2)), 0.3
    psi = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
    psi[0] *= 1e18
    psi[:, 0] *= 1e18
    p = np.maximum(abs(psi.real), abs(psi.imag))
    c = np.exp(mu)
    near = [m * p] + [np.roll(p, s, ax) * (c if ax == 0 else 1) for ax in (0, 1) for s in (-1, 1)]
    for ax in (0, 1):
        if bc[ax] == 0:   # s = -1 brings in the next site, whose link is open on the last slice; s = 1 the previous
            edge = [slice(None)] * 2
            for s, at in ((-1, -1), (1, 0)):
                edge[ax] = at
                near[1 + 2 * ax + (s > 0)][tuple(edge)] = 0
    S = np.maximum.reduce(near)
    o = oracle_lib.Oracle(nt, nx, m, 0.5, mu, *bc)
    with tg.Lattice(nt, nx, m, 0.5, mu, *bc) as L:
        L.set_gauge(A)
        for got, want in ((L.fm_mul(psi), o.M(A, psi)), (L.fm_conjugate_mul(psi), o.Mdag(A, psi))):
            d = got - want
            assert np.all(np.maximum(abs(d.real), abs(d.imag)) <= 50 * 2.0 ** -53 * S)
        x, res = L.fmdm_invert_cg(psi, tg.cg_params(rel_tol=1e-10, abs_tol2=0))
        assert res.status == 0
        assert np.linalg.norm(psi - o.Mdag(A, o.M(A, x))) <= 1.5e-10 * np.linalg.norm(psi)
