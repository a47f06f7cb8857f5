"""FP64 batches of different chains in several threads at once: their launches need
different amounts of shared memory, and no batch may change what another's launch is
allowed."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("instance", [51201, 25604, 1451241])
def test_batches_in_threads(instance):
    import thirring2d_gb300 as tg
    sides, runs = (24, 48, 26, 47, 28, 46, 30, 45), 1500
    bp = tg.batch_params(nsteps=1, tau=0.02, block=instance, use_graph=False, cg=tg.cg_params(rel_tol=0.5, abs_tol2=0))
    errors, fields = [], {}

    def batch(side):
        return tg.Batch([dict(nt=side, nx=side, m=3.0, g=0.7, mu=0.0, bc_t=-1, bc_x=1, seed=side)])

    def work(side):
        try:
            B = batch(side)
            for _ in range(runs):
                B.trajectory(bp)
            fields[side] = B.get_gauge(0)
            B.close()
        except Exception as e:  # noqa: BLE001  (reported below: a thread's exception ends only the thread)
            errors.append((side, repr(e)))
    threads = [threading.Thread(target=work, args=(s,)) for s in sides]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    B = batch(sides[1])    # and every batch ran what it runs alone
    for _ in range(runs):
        B.trajectory(bp)
    assert np.array_equal(B.get_gauge(0), fields[sides[1]])
    B.close()
