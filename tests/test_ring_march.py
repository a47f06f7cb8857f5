"""The prefetched FP64 march (march_ring64 in csrc/tg_stencil.cuh), audited on the
CPU: its index arithmetic restated, every row and edge a step reads must be in
the ring when it is read (its group waited for, not yet overwritten), and every
address fetched must lie inside the lattice and be the one the step needs."""
import pytest

K = 4  # kMarchT, and rows of the ring


def run(nt, nx, xw, ta, tb):
    n, x0 = tb - ta, xw * 32
    xle, xre = (nx - 1 if x0 == 0 else x0 - 1), (0 if x0 + 32 == nx else x0 + 32)
    slots, edges = [None] * K, [None, None]   # what each holds: (row, group)
    groups, written = 0, []

    def issue(i, slot):
        t = ta + i
        tp = 0 if t + 1 == nt else t + 1
        for a in (tp * nx + x0, tp * nx + x0 + 31, t * nx + x0 + 31):
            assert 0 <= a < nt * nx
        slots[slot] = (i, groups, tp)
        if i % K == 0:
            rows = [min(t + (lane & (K - 1)), tb - 1) for lane in range(2 * K)]
            assert all(ta <= r < tb for r in rows)
            edges[(i // K) & 1] = (i // K, groups, [(r, xle if lane < K else xre) for lane, r in enumerate(rows)])

    for i in range(K - 1):
        if i < n:
            issue(i, i)
        groups += 1
    ef = None
    for i0 in range(0, n, K):
        for ic in range(K):
            i = i0 + ic
            if i >= n:
                break
            if i + K - 1 < n:
                issue(i + K - 1, (ic + K - 1) % K)
            groups += 1
            done = groups - (K - 1)           # wait_group K-1: all groups but the last K-1
            if ic == 0:
                chunk, grp, ef = edges[(i0 // K) & 1]
                assert chunk == i0 // K and grp < done
            row, grp, tp = slots[ic]
            assert row == i and grp < done and tp == (ta + i + 1) % nt
            assert ef[ic] == (ta + i, xle) and ef[K + ic] == (ta + i, xre)
            written.append(ta + i)
    assert written == list(range(ta, tb))


@pytest.mark.parametrize("nt,nx", [(4, 32), (8, 64), (64, 32), (128, 96)])
def test_every_segment(nt, nx):
    for xw in range(nx // 32):
        for ta in range(nt):
            for tb in {ta + 1, ta + 2, min(ta + 5, nt), min(ta + 13, nt), nt}:
                if ta < tb <= nt:
                    run(nt, nx, xw, ta, tb)
