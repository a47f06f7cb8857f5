"""The on-chip CG of small lattices (csrc/tg_cluster_cg.cu): against the oracle's CG
at the sizes where its split can go wrong -- a site per block, rows fewer than
blocks, odd sides, windows that wrap onto their own block, several sites per
thread, the largest lattice of each precision -- and on right-hand sides and masses that leave
the integer sums' scale."""
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


SHAPES = [(2, 2), (2, 64), (3, 5), (8, 8), (5, 100), (16, 16), (17, 31), (33, 24), (60, 100), (64, 64), (128, 128)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mu", [0.0, 0.2])
@pytest.mark.parametrize("nt,nx", SHAPES + [(256, 256)])
def test_solution_against_oracle(tg, oracle_lib, monkeypatch, nt, nx, mu, precision):
    """CG to 1e-11 relative from the same start: two solutions whose residuals are
    1e-11 of b differ by at most 2e-11 / m of |x| in the worst direction; m = 0.3.
    The FP64 iteration count is the oracle's; the mixed one the grid solver's, whose
    recurrences and reliable updates it shares (on a lattice of a few sites
    either restarts a CG that would have ended exactly)."""
    if precision == 0 and nt * nx > 128 * 128:
        pytest.skip("the mixed solver's largest case")
    rng = np.random.default_rng(nt * 1000 + nx)
    A, b, m = rng.normal(0, 0.5, (nt, nx, 2)), cplx(rng, (nt, nx)), 0.3
    o = oracle_lib.Oracle(nt, nx, m, 0.5, mu, -1, 1)
    xo, st, it = o.cg(A, b, rel_tol=1e-11, abs_tol2=0)
    cp = tg.cg_params(rel_tol=1e-11, abs_tol2=0, precision=precision)
    with tg.Lattice(nt, nx, m, 0.5, mu, -1, 1) as L:
        L.set_gauge(A)
        x, res = L.fmdm_invert_cg(b, cp)
        y, _ = L.fmdm_invert_cg(b, cp)
    if precision == 1:
        monkeypatch.setenv("TG_CLUSTER_CG", "0")
        with tg.Lattice(nt, nx, m, 0.5, mu, -1, 1) as L:
            L.set_gauge(A)
            it = L.fmdm_invert_cg(b, cp)[1].iterations
    assert res.status == 0 and st == 0
    assert rel(x, xo) < 2e-11 / m * 2
    assert abs(res.iterations - it) <= max(2, it // 20)
    assert np.linalg.norm(b - o.Mdag(A, o.M(A, x))) <= 1.5e-11 * np.linalg.norm(b)
    assert np.array_equal(x, y)


@pytest.mark.parametrize("blocks,threads", [(1, 32), (1, 512), (2, 96), (4, 256), (8, 64), (16, 32), (16, 512)])
@pytest.mark.parametrize("precision", [0, 1])
def test_shapes_agree(tg, monkeypatch, blocks, threads, precision):
    """Every cluster shape against the grid solver on one lattice: the same system to
    1e-11, the rounding of sums apart."""
    nt, nx, m = 20, 36, 0.2
    rng = np.random.default_rng(4)
    A, b = rng.normal(0, 0.5, (nt, nx, 2)), cplx(rng, (nt, nx))
    out = []
    for v in ("0", f"{blocks}:{threads}"):
        monkeypatch.setenv("TG_CLUSTER_CG", v)
        with tg.Lattice(nt, nx, m, 0.5, 0.1, -1, -1) as L:
            L.set_gauge(A)
            out.append(L.fmdm_invert_cg(b, tg.cg_params(rel_tol=1e-11, abs_tol2=0, precision=precision)))
    assert out[0][1].status == out[1][1].status == 0
    assert rel(out[1][0], out[0][0]) < 4e-11 / m


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", ["heavy", "light", "point", "tiny", "large"])
def test_sums_that_leave_their_scale(tg, oracle_lib, case, precision):
    nt, nx = 24, 40
    m = {"heavy": 50.0, "light": 0.02}.get(case, 0.2)
    rng = np.random.default_rng(12)
    A = rng.normal(0, 0.4, (nt, nx, 2))
    b = cplx(rng, (nt, nx)) * {"tiny": 1e-9, "large": 1e9}.get(case, 1.0)
    if case == "point":
        b = np.zeros((nt, nx), complex)
        b[3, 5] = 1.0
    o = oracle_lib.Oracle(nt, nx, m, 0.5, 0.0, -1, 1)
    with tg.Lattice(nt, nx, m, 0.5, 0.0, -1, 1) as L:
        L.set_gauge(A)
        x, res = L.fmdm_invert_cg(b, tg.cg_params(rel_tol=1e-10, abs_tol2=0, precision=precision))
    assert res.status == 0
    assert np.linalg.norm(b - o.Mdag(A, o.M(A, x))) <= 1.5e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("precision", [0, 1])
def test_edge_cases(tg, precision):
    """b = 0, the iteration cap, NaN, and a singular operator: the statuses of the grid solver."""
    rng = np.random.default_rng(9)
    with tg.Lattice(12, 20, 0.3, 0.5, 0.0, -1, 1) as L:
        L.set_gauge(rng.normal(0, 0.5, (12, 20, 2)))
        b = cplx(rng, (12, 20))
        x, res = L.fmdm_invert_cg(np.zeros((12, 20), complex), tg.cg_params(precision=precision))
        assert res.status == 0 and res.iterations == 0 and not x.any()
        x, res = L.fmdm_invert_cg(b, tg.cg_params(maxiter=3, precision=precision))
        assert res.status == tg.native.TG_E_NOCONV and res.iterations == 3
        bad = b.copy()
        bad[2, 3] = np.nan
        x, res = L.fmdm_invert_cg(bad, tg.cg_params(precision=precision))
        assert res.status == tg.native.TG_E_NAN
        x, res = L.fmdm_invert_cg(b, tg.cg_params(rel_tol=1e-10, abs_tol2=0, precision=precision))
        assert res.status == 0
    with tg.Lattice(8, 8, 0.0, 0.5, 0.0, 1, 1) as L:
        x, res = L.fmdm_invert_cg(cplx(rng, (8, 8)), tg.cg_params(rel_tol=1e-12, abs_tol2=0, maxiter=5000,
                                                                  precision=precision))
        assert res.status in (tg.native.TG_E_DIVERGED, tg.native.TG_E_NAN, tg.native.TG_E_NOCONV)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nt,nx", [(16, 16), (48, 64), (128, 128)])
def test_grid_solver_on_small_lattices(tg, oracle_lib, monkeypatch, nt, nx, precision):
    """The grid solver stays what runs when the cluster one is turned off."""
    monkeypatch.setenv("TG_CLUSTER_CG", "0")
    test_solution_against_oracle(tg, oracle_lib, monkeypatch, nt, nx, 0.0, precision)


@pytest.mark.parametrize("scale", [1e-8, 3e-9, 1e-9, 3e-10])
def test_mixed_residuals_whose_squares_are_denormal(tg, oracle_lib, scale):
    """r^2 per site falls below 2^-126 in FP32 near the end of the solve."""
    nt, nx, m = 24, 40, 0.3
    rng = np.random.default_rng(2)
    A, b = rng.normal(0, 0.5, (nt, nx, 2)), cplx(rng, (nt, nx)) * scale
    o = oracle_lib.Oracle(nt, nx, m, 0.5, 0.0, -1, 1)
    with tg.Lattice(nt, nx, m, 0.5, 0.0, -1, 1) as L:
        L.set_gauge(A)
        x, res = L.fmdm_invert_cg(b, tg.cg_params(rel_tol=1e-11, abs_tol2=0, precision=1))
    assert res.status == 0
    assert np.linalg.norm(b - o.Mdag(A, o.M(A, x))) <= 1.5e-11 * np.linalg.norm(b)


# the largest lattices that the cluster takes and the next ones, which the grid's shared memory does:
# 16 blocks of 512 sites in FP64, of 2400 mixed; and the cluster's own limit with the grid's turned off
@pytest.mark.parametrize("nt,nx,precision,env", [(90, 91, 0, {}), (91, 91, 0, {}), (64, 128, 0, {}), (195, 196, 1, {}), (196, 196, 1, {}),
                                                 (120, 320, 1, {}), (113, 120, 0, {"TG_GRID_CG": "0"}), (220, 240, 1, {"TG_GRID_CG": "0"})])
def test_hand_over_to_the_grid(tg, oracle_lib, monkeypatch, nt, nx, precision, env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    test_solution_against_oracle(tg, oracle_lib, monkeypatch, nt, nx, 0.0, precision)
