"""The FP64 operator on the integer pipes, on the GPU: both stencil paths on
operands of very different sizes and on operands that are not finite, against
the oracle's FP64 operator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import thirring2d_gb300 as tg
    tg.native.load()
    return tg


def scale(psi, m, mu):
    """Per site: the largest |part| among the five operands, times its constant."""
    p = np.maximum(abs(psi.real), abs(psi.imag))
    c = np.exp(abs(mu))
    return np.maximum.reduce([abs(m) * p] + [c * np.roll(p, s, 0) for s in (1, -1)] + [np.roll(p, s, 1) for s in (1, -1)])


@pytest.mark.parametrize("nt,nx,mu,m", [(2, 2, 0.0, 0.3), (3, 5, 0.2, 0.1), (8, 32, 0.0, 0.05), (7, 64, 0.1, 0.5),
                                        (12, 96, 0.0, 0.0), (64, 32, 0.3, 2.0), (6, 33, 0.0, 0.1), (128, 160, 0.0, 0.02)])
@pytest.mark.parametrize("spread", [0, 12])
def test_operator_against_oracle(tg, oracle_lib, nt, nx, mu, m, spread):
    """Within 5 * 2^-53 of the site's scale for the integer form, and the oracle's
    own 18 roundings of at most 5 scales: 5 + 18 * 5 / 2 = 50 of 2^-53."""
    rng = np.random.default_rng(nt * 1000 + nx + spread)
    A = rng.normal(0, 0.7, (nt, nx, 2))
    psi = (rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))) * 10.0 ** rng.integers(-spread, spread + 1, (nt, nx))
    o = oracle_lib.Oracle(nt, nx, m, 0.5, mu, -1, 1)
    with tg.Lattice(nt, nx, m, 0.5, mu, -1, 1) as L:
        L.set_gauge(A)
        S = scale(psi, m, mu)
        for got, want in ((L.fm_mul(psi), o.M(A, psi)), (L.fm_conjugate_mul(psi), o.Mdag(A, psi))):
            d = got - want
            assert np.all(np.maximum(abs(d.real), abs(d.imag)) <= 50 * 2.0 ** -53 * S)


@pytest.mark.parametrize("nt,nx", [(8, 32), (6, 10)])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e305, 1e-310, 0.0])
def test_extreme_operands(tg, oracle_lib, nt, nx, value):
    """One extreme site in an ordinary vector, and a vector of nothing else: the
    same sites are finite as in FP64, and zero stays zero."""
    rng = np.random.default_rng(5)
    A = rng.normal(0, 0.7, (nt, nx, 2))
    o = oracle_lib.Oracle(nt, nx, 0.1, 0.5, 0.0, -1, 1)
    one = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
    one[nt // 2, nx // 2] = complex(value, 1.0)
    with tg.Lattice(nt, nx, 0.1, 0.5, 0.0, -1, 1) as L, np.errstate(all="ignore"):
        L.set_gauge(A)
        for psi in (one, np.full((nt, nx), complex(value, 0.0))):
            for got, want in ((L.fm_mul(psi), o.M(A, psi)), (L.fm_conjugate_mul(psi), o.Mdag(A, psi))):
                assert np.array_equal(np.isfinite(got), np.isfinite(want))
                ok = np.isfinite(want)
                assert np.allclose(got[ok], want[ok], rtol=1e-12, atol=1e-12 * np.abs(np.nan_to_num(psi[np.isfinite(psi)])).max(initial=0.0) + 1e-320)


def test_gauge_field_that_is_not_finite(tg):
    """A NaN or Inf link makes the sites it touches NaN, as cos and sin of it do."""
    rng = np.random.default_rng(6)
    for nt, nx in ((8, 32), (6, 10)):
        A = rng.normal(0, 0.7, (nt, nx, 2))
        A[2, 3, 0], A[4, 5, 1] = np.nan, np.inf
        psi = rng.normal(size=(nt, nx)) + 1j * rng.normal(size=(nt, nx))
        bad = np.zeros((nt, nx), bool)
        bad[2, 3] = bad[3, 3] = bad[4, 5] = bad[4, 6] = True
        with tg.Lattice(nt, nx, 0.1, 0.5, 0.0, -1, 1) as L:
            L.set_gauge(A)
            for out in (L.fm_mul(psi), L.fm_conjugate_mul(psi)):
                assert np.array_equal(np.isnan(out), bad)
            x, res = L.fmdm_invert_cg(psi)
            assert res.status == tg.native.TG_E_NAN


@pytest.mark.parametrize("nt,nx,mu", [(8, 32, 0.0), (6, 10, 0.0), (40, 70, 0.2), (64, 64, 0.0)])
@pytest.mark.parametrize("value", [1.0, 0.0, -0.0, 1e-310])
def test_vectors_that_are_zero_but_for_one_site(tg, oracle_lib, nt, nx, mu, value):
    """M and M^dagger of a point source: the five sites it reaches, to rounding (18 of 2^-53
    and the integer form's 5, of the value; denormals have steps of 2^-1074 instead), and zeros;
    the solve's residual meets the tolerance 1e-11 (and rounding) where there is one."""
    rng = np.random.default_rng(7)
    A = rng.normal(0, 0.7, (nt, nx, 2))
    psi = np.zeros((nt, nx), complex)
    psi[nt // 2, nx - 1] = complex(value, 0.0)
    o = oracle_lib.Oracle(nt, nx, 0.3, 0.5, mu, -1, 1)
    with tg.Lattice(nt, nx, 0.3, 0.5, mu, -1, 1) as L:
        L.set_gauge(A)
        for got, want in ((L.fm_mul(psi), o.M(A, psi)), (L.fm_conjugate_mul(psi), o.Mdag(A, psi))):
            assert np.array_equal(got == 0, want == 0)
            assert np.abs(got - want).max() <= 50 * 2.0 ** -53 * abs(value) + 20 * 2.0 ** -1074
        if value == 1.0:
            x, res = L.fmdm_invert_cg(psi, tg.cg_params(rel_tol=1e-11, abs_tol2=0))
            assert res.status == 0
            assert np.linalg.norm(psi - o.Mdag(A, o.M(A, x))) <= 1.5e-11
