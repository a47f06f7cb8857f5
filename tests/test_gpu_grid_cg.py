"""The on-chip CG of middle-sized lattices (csrc/tg_grid_cg.cu) against the oracle's CG
where its split can go wrong: one block, blocks shorter than a row (every site is a
neighbour's), ragged shares, several sites per thread, the largest lattice of each
precision, and sums that leave their scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import thirring2d_gb300 as tg
    tg.native.load()
    return tg


def cplx(rng, shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def solve(tg, oracle, nt, nx, m, mu, precision, b_scale=1.0):
    """Both solutions' residuals are 1e-11 of b: they differ by at most 2e-11 / m of |x|
    (doubled for the rounding of sums)."""
    rng = np.random.default_rng(nt * 1000 + nx)
    A, b = rng.normal(0, 0.5, (nt, nx, 2)), cplx(rng, (nt, nx)) * b_scale
    o = oracle.Oracle(nt, nx, m, 0.5, mu, -1, 1)
    xo, st, it = o.cg(A, b, rel_tol=1e-11, abs_tol2=0)
    cp = tg.cg_params(rel_tol=1e-11, abs_tol2=0, precision=precision)
    with tg.Lattice(nt, nx, m, 0.5, mu, -1, 1) as L:
        L.set_gauge(A)
        x, res = L.fmdm_invert_cg(b, cp)
        y, _ = L.fmdm_invert_cg(b, cp)
    assert res.status == 0 and st == 0
    assert rel(x, xo) < 2e-11 / m * 2
    if precision == 0:
        assert abs(res.iterations - it) <= max(2, it // 20)
    assert np.linalg.norm(b - o.Mdag(A, o.M(A, x))) <= 1.5e-11 * np.linalg.norm(b)
    assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nt,nx,shape,mu", [
    (2, 64, "1:32", 0.0), (3, 5, "1:512", 0.2), (16, 16, "3:32", 0.2), (12, 200, "37:64", 0.2), (12, 200, "37:32", 0.0),
    (33, 24, "5:96", 0.0), (64, 64, "64:64", 0.2), (100, 60, "7:256", 0.0), (64, 64, "4:512", 0.2)])
def test_shapes_against_oracle(tg, oracle_lib, monkeypatch, nt, nx, shape, mu, precision):
    monkeypatch.setenv("TG_CLUSTER_CG", "0")
    monkeypatch.setenv("TG_GRID_CG", shape)
    solve(tg, oracle_lib, nt, nx, 0.3, mu, precision)


@pytest.mark.parametrize("nt,nx,shape,mu", [
    (2, 64, "1:32:1", 0.0), (3, 6, "1:480:1", 0.2), (2, 2, "1:32:1", 0.0), (16, 16, "3:32:1", 0.2), (12, 200, "37:64:1", 0.2), (33, 24, "5:96:1", 0.0),
    (100, 60, "7:256:1", 0.0), (64, 64, "4:480:1", 0.2), (96, 100, "3:480:1", 0.0), (131, 190, "152:480:1", 0.2)])
def test_links_from_global_memory_against_oracle(tg, oracle_lib, monkeypatch, nt, nx, shape, mu):
    monkeypatch.setenv("TG_CLUSTER_CG", "0")
    monkeypatch.setenv("TG_GRID_CG", shape)
    solve(tg, oracle_lib, nt, nx, 0.3, mu, 1)


@pytest.mark.parametrize("nt,nx,shape,mu", [
    (2, 64, "1:32:2", 0.0), (2, 2, "1:32:2", 0.0), (12, 200, "37:64:2", 0.2), (33, 24, "5:96:2", 0.0), (100, 60, "7:256:2", 0.0),
    (64, 64, "4:512:2", 0.2), (131, 190, "152:512:2", 0.2)])
def test_pairs_of_sites_against_oracle(tg, oracle_lib, monkeypatch, nt, nx, shape, mu):
    monkeypatch.setenv("TG_CLUSTER_CG", "0")
    monkeypatch.setenv("TG_GRID_CG", shape)
    solve(tg, oracle_lib, nt, nx, 0.3, mu, 1)


@pytest.mark.parametrize("nt,nx,mu,precision", [(128, 256, 0.0, 0), (131, 190, 0.2, 0), (256, 256, 0.2, 0), (400, 400, 0.0, 0),
                                                (256, 300, 0.0, 1), (512, 512, 0.2, 1), (700, 701, 0.0, 1),
                                                (1001, 902, 0.2, 1), (1024, 1024, 0.0, 1)])
def test_middle_sizes_against_oracle(tg, oracle_lib, nt, nx, mu, precision):
    solve(tg, oracle_lib, nt, nx, 0.3, mu, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", ["heavy", "tiny", "large"])
def test_sums_that_leave_their_scale(tg, oracle_lib, monkeypatch, case, precision):
    monkeypatch.setenv("TG_CLUSTER_CG", "0")
    monkeypatch.setenv("TG_GRID_CG", "9:96")
    solve(tg, oracle_lib, 24, 40, 50.0 if case == "heavy" else 0.3, 0.0, precision,
          {"tiny": 1e-9, "large": 1e9}.get(case, 1.0))


@pytest.mark.parametrize("precision", [0, 1])
def test_edge_cases(tg, precision):
    """b = 0, the iteration cap and NaN: the statuses of the other solvers."""
    nt, nx = 256, 320
    rng = np.random.default_rng(9)
    with tg.Lattice(nt, nx, 0.3, 0.5, 0.0, -1, 1) as L:
        L.set_gauge(rng.normal(0, 0.5, (nt, nx, 2)))
        b = cplx(rng, (nt, nx))
        x, res = L.fmdm_invert_cg(np.zeros((nt, nx), complex), tg.cg_params(precision=precision))
        assert res.status == 0 and res.iterations == 0 and not x.any()
        x, res = L.fmdm_invert_cg(b, tg.cg_params(maxiter=3, precision=precision))
        assert res.status == tg.native.TG_E_NOCONV and res.iterations == 3
        b[2, 3] = np.nan
        x, res = L.fmdm_invert_cg(b, tg.cg_params(precision=precision))
        assert res.status == tg.native.TG_E_NAN
