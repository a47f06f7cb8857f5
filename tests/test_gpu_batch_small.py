"""FP64 chains that one block solves in its shared memory (block_cg64_small in
csrc/tg_batch_impl.cuh): every chain reproduces the single-lattice trajectory
with the same seed, on the instances that differ in what they keep there, at
sizes up to and past their share, odd sides among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tg():
    import thirring2d_gb300 as tg
    tg.native.load()
    return tg


@pytest.mark.parametrize("instance", [12808, 25604, 25602, 51201, 1451241])
@pytest.mark.parametrize("sizes", [[(8, 8), (11, 12), (16, 16), (17, 15)], [(16, 16), (24, 24), (32, 32), (3, 50)],
                                   [(48, 48), (47, 49), (12, 128)], [(64, 64), (16, 16)]])
def test_chains_match_single_lattices(tg, instance, sizes):
    """dH to 1e-8 (solves to 1e-12; the two paths' sums are added in different orders),
    the same decisions, fields to 1e-9 after two trajectories of stable steps."""
    rng = np.random.default_rng(17)
    chains = [dict(nt=t, nx=x, m=0.3, g=0.7, mu=0.1 * (k % 2), bc_t=-1, bc_x=1 - 2 * (k % 2), seed=40 + k)
              for k, (t, x) in enumerate(sizes)]
    A0 = [rng.normal(0, 0.2, (t, x, 2)) for t, x in sizes]
    cg = tg.cg_params(rel_tol=1e-12, abs_tol2=0.0)
    B = tg.Batch(chains)
    for i, A in enumerate(A0):
        B.set_gauge(i, A)
    res = [B.trajectory(tg.batch_params(nsteps=4, tau=0.1, block=instance, cg=cg)) for _ in range(2)]
    for i, c in enumerate(chains):
        with tg.Lattice(c["nt"], c["nx"], c["m"], c["g"], c["mu"], c["bc_t"], c["bc_x"]) as L:
            L.set_gauge(A0[i])
            hp = tg.hmc_params(nsteps=4, tau=0.1, rng=tg.native.RNG_PHILOX, seed=c["seed"], cg=cg)
            for k in range(2):
                r, b = L.update_gauge(hp), res[k][i]
                assert b.status == 0 and r.status == 0 and b.accepted == r.accepted
                assert abs(b.dH - r.dH) <= 1e-8 * max(1.0, abs(r.dH))
                assert abs(b.cg_iterations - r.cg_iterations) <= 2 * r.cg_solves
            assert np.abs(B.get_gauge(i) - L.get_gauge()).max() < 1e-9
    B.close()


@pytest.mark.parametrize("instance", [12808, 25604])
@pytest.mark.parametrize("precision", [0, 1])
def test_instances_with_a_kernel_per_precision(tg, instance, precision):
    """The 64-register instances run mixed solves, and FP64 ones on other kernels: both
    follow the 512-thread instance (dH to 1e-7 with solves to 1e-11, the same decisions)."""
    rng = np.random.default_rng(18)
    chains = [dict(nt=t, nx=x, m=0.3, g=0.7, mu=0.1 * (k % 2), bc_t=-1, bc_x=1, seed=60 + k)
              for k, (t, x) in enumerate([(8, 8), (16, 16), (17, 15), (32, 32), (30, 64), (64, 64)])]
    A0 = [rng.normal(0, 0.2, (c["nt"], c["nx"], 2)) for c in chains]
    out = []
    for inst in (51201, instance):
        B = tg.Batch(chains)
        for i, A in enumerate(A0):
            B.set_gauge(i, A)
        out.append(B.trajectory(tg.batch_params(nsteps=4, tau=0.1, block=inst,
                                                cg=tg.cg_params(rel_tol=1e-11, abs_tol2=0.0, precision=precision))))
        B.close()
    for a, b in zip(*out):
        assert a.status == b.status == 0 and a.accepted == b.accepted
        assert abs(a.dH - b.dH) <= 1e-7 * max(1.0, abs(a.dH))
