"""Column marches whose last strip is not full: the operator in both precisions, bit for bit
against one site per thread, and solves (two-sum and single-reduction mixed, FP64)
against that path's, at widths around the strip's and row counts around the
chunk's."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import thirring2d_gb300 as tg
    tg.native.load()
    return tg


def both(monkeypatch, f):
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("TG_MARCH", flag)
        out.append(f())
    return out


@pytest.mark.parametrize("nt,nx", [(2, 29), (3, 30), (5, 31), (6, 58), (7, 63), (4, 90), (9, 95), (13, 126), (10, 300), (33, 1000)])
@pytest.mark.parametrize("mu", [0.0, 0.2])
def test_operator_equals_site_path(tg, monkeypatch, nt, nx, mu):
    rng = np.random.default_rng(nt * 1000 + nx)
    A = rng.normal(0, 0.6, (nt, nx, 2))
    psi = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
    p32 = torch.from_numpy(psi).to("cuda", torch.complex64)

    def run():
        with tg.Lattice(nt, nx, 0.2, 0.5, mu, -1, 1) as L:
            L.set_gauge(A)
            o32 = [torch.empty_like(p32) for _ in range(2)]
            torch.cuda.synchronize()
            for d in (0, 1):
                L.apply_dev(p32.data_ptr(), o32[d].data_ptr(), bool(d), tg.native.PREC_MIXED)
            L.synchronize()
            return L.fm_mul(psi), L.fm_conjugate_mul(psi), o32[0].cpu().numpy(), o32[1].cpu().numpy(), L.stochastic_md_action(psi)
    m, s = both(monkeypatch, run)
    for a, b in zip(m[:2], s[:2]):
        assert np.array_equal(a, b)
    for a, b in zip(m[2:4], s[2:4]):  # the compiler may contract the two paths' FP32 sums differently
        assert np.abs(a - b).max() <= 2.0 ** -21 * np.abs(b).max()
    assert abs(m[4] - s[4]) <= 1e-12 * abs(s[4])


@pytest.mark.parametrize("nt,nx", [(5, 31), (7, 63), (9, 95), (40, 300), (45, 301)])
@pytest.mark.parametrize("form", ["fp64", "twosum", "onesum"])
def test_solves_equal_site_path(tg, monkeypatch, nt, nx, form):
    """The grid solvers on the march (TG_PCG_BLOCK keeps it at small sizes) and site by
    site: both residuals are 1e-11 of b, so solutions differ by 4e-11 / m at most."""
    rng = np.random.default_rng(nx)
    A, m = rng.normal(0, 0.4, (nt, nx, 2)), 0.2
    b = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
    cp = tg.cg_params(rel_tol=1e-11, abs_tol2=0, precision=0 if form == "fp64" else 1)

    def run(**env):
        for k in ("TG_PCG_BLOCK", "TG_MIXED_CG", "TG_MARCH", "TG_CLUSTER_CG"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        with tg.Lattice(nt, nx, m, 0.5, 0.1, -1, -1) as L:
            L.set_gauge(A)
            return L.fmdm_invert_cg(b, cp)
    ref, r0 = run(TG_MARCH="0", TG_CLUSTER_CG="0")
    x, r1 = run(TG_PCG_BLOCK="512") if form == "fp64" else run(TG_PCG_BLOCK="512", TG_MIXED_CG=form)
    assert r0.status == r1.status == 0
    assert np.linalg.norm(x - ref) <= 4e-11 / m * np.linalg.norm(ref)
