"""The tiled particle layout (rows sized for a group's mean lane, the excess of
fuller cells in other lanes' free slots) against the slot-order push, where it
can go wrong: crowded and empty cells, ragged sides, groups that outgrow their
rows between two full sorts."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION, Pic3D, PicConfig, PicError
from util import rel_norm

pytestmark = pytest.mark.gpu


def crowd(n, rng, speed):
    """Rows over an (nx, ny, nz) grid: a few cells with up to 300 particles
    (one of them the last lane of the last group), a thin background; all
    drifting along x at `speed`, so that at 0.9 they leave their columns
    within six steps."""
    cells = [tuple(2 + int(rng.integers(m)) for m in n) for _ in range(6)]
    cells.append(tuple(m + 1 for m in n))
    xyz = [np.array(c) + rng.random((k, 3)) for c, k in zip(cells, (300, 100, 33, 32, 31, 1, 65))]
    xyz.append(2 + rng.random((40, 3)) * np.array(n))
    xyz = np.concatenate(xyz)
    v = rng.normal(0, 0.02, xyz.shape) + [speed, 0, 0.05]
    return np.column_stack([xyz, v, np.full(len(xyz), 0.01 / 4)])


def context(n, precision, slot_order):
    P = Pic3D(PicConfig.normalized(*n, 4, precision=precision, diag_every_step=0, sort_interval=1,
                                   add_interval=1000, slot_order=slot_order, capacity=200000))
    P.init_grid()
    return P


def ordered(rows):
    return rows[np.lexsort(rows.T[::-1])]


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [(8, 8, 8), (5, 7, 31), (6, 5, 33), (9, 6, 64)])
@pytest.mark.parametrize("speed", [0.1, 0.9])
def test_layout_keeps_particles_and_their_sums(n, speed, precision):
    rng = np.random.default_rng(sum(n) + int(10 * speed))
    rows = [crowd(n, rng, speed) for _ in range(2)]
    with context(n, precision, 0) as T, context(n, precision, 1) as S:
        for s in (ION, ELECTRON):
            T.set_particles(s, rows[s])
            S.set_particles(s, rows[s])
        T.sorting()
        for s in (ION, ELECTRON):  # a sort moves records, bit for bit
            assert np.array_equal(ordered(T.particles(s)), ordered(S.particles(s)))
        for _ in range(8):  # a re-layout in every second step or so
            T.step(1)
            S.step(1)
            if precision == 64:  # each step rounds a value a few times: 8 steps stay within 1e-12 of it
                g, h = T.grid(), S.grid()
                for q in range(18):
                    assert rel_norm(g[..., q], h[..., q]) < 1e-11 or np.abs(g[..., q] - h[..., q]).max() < 1e-15
        for s in (ION, ELECTRON):
            a, b = T.particles(s), S.particles(s)
            assert len(a) == len(b)
            if precision == 64:
                assert rel_norm(ordered(np.round(a, 9)), ordered(np.round(b, 9))) < 1e-8
        assert T.status()[0] == 0


@pytest.mark.parametrize("case", ["long moves", "ballistic at 3 c", "ballistic at 9 c", "wraps"])
def test_particles_off_the_short_path(case):
    """Moves of a cell and more per half step, ballistic particles that Boris
    has not slowed, and more particles wrapped round the x faces than a warp's
    list holds: the tiled push hands them to the general one (FP64; a step
    rounds a value a few times, so 1e-11 covers three)."""
    n = (12, 9, 40)
    kw = {"long moves": dict(dt=2.5), "wraps": {}}.get(case, dict(absorb_grid2=5))
    speed = {"ballistic at 3 c": 3.0, "ballistic at 9 c": 9.0, "wraps": 0.95}.get(case, 0.3)
    rng = np.random.default_rng(len(case))
    xyz = 2 + rng.random((6000, 3)) * np.array(n)
    if case == "wraps":
        xyz[:, 0] = n[0] + 1 + rng.random(6000)
        xyz[:, 1] = 3 + rng.random(6000)
    v = rng.normal(0, 0.1 * speed, xyz.shape) + [0.9 * speed, 0, 0.1]
    if case == "wraps":
        v[:] = [0.94, 0, 0.05]
    rows = np.column_stack([xyz, v, np.full(len(xyz), 0.01 / 4)])
    P = []
    for slot_order in (0, 1):
        P.append(Pic3D(PicConfig.normalized(*n, 4, precision=64, diag_every_step=0, sort_interval=1000,
                                            add_interval=1000, slot_order=slot_order, capacity=200000, **kw)))
        P[-1].init_grid()
        for s in (ION, ELECTRON):
            P[-1].set_particles(s, rows)
    for _ in range(3 if case != "wraps" else 8):
        for p in P:
            p.step(1)
        g, h = P[0].grid(), P[1].grid()
        for q in range(18):
            assert rel_norm(g[..., q], h[..., q]) < 1e-11 or np.abs(g[..., q] - h[..., q]).max() < 1e-15
    for s in (ION, ELECTRON):
        a, b = P[0].particles(s), P[1].particles(s)
        assert len(a) == len(b) and rel_norm(ordered(np.round(a, 8)), ordered(np.round(b, 8))) < 1e-7
    (ra, ca), (rb, cb) = P[0].status(), P[1].status()
    assert ra == rb and np.array_equal(ca, cb)
    for p in P:
        p.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [(9, 8, 33), (10, 9, 64)])
def test_single_functions_over_the_layout(n, precision):
    """The push and drift loops called by themselves on a sorted store with a
    refill behind the layout, against the same calls in slot order. FP64: 1e-11
    as above. FP32: a step's velocities differ by the square roots' and
    divisions' roundings (2e-7 each, a few of them: 2e-6), the sums of 8 to 300
    such terms by as much."""
    rng = np.random.default_rng(n[0])
    rows = [crowd(n, rng, 0.2) for _ in range(2)]
    P = [context(n, precision, slot_order) for slot_order in (0, 1)]
    for p in P:
        for s in (ION, ELECTRON):
            p.set_particles(s, rows[s])
        p.sorting()
        p.add_flat()
        for step in range(2):
            p.renew_grid()
            p.renew_b4_2()
            if step == 0:
                p.push_deposit_j()
            else:  # one species at a time, the second first
                p.push_deposit_j(ELECTRON)
                p.push_deposit_j(ION)
            p.renew_b4_2()
            p.drift_deposit_n()
            p.reduce_current()
            p.renew_e4_2()
            p.sr_particle()
    g, h = P[0].grid(), P[1].grid()
    tol = 1e-11 if precision == 64 else 1e-5
    for q in range(18):
        assert rel_norm(g[..., q], h[..., q]) < tol or np.abs(g[..., q] - h[..., q]).max() < 1e-15
    for s in (ION, ELECTRON):
        assert P[0].particle_count(s) == P[1].particle_count(s)
    (ra, ca), (rb, cb) = P[0].status(), P[1].status()
    assert ra == rb == 0 and np.array_equal(ca, cb)
    for p in P:
        p.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_hand_over_without_append_slots(precision):
    """Particles that change lanes while the buffer ends with the layout: a
    crowd moves into a cell whose lane has fewer holes than arrivals, and no
    slot is left outside the layout. None may be lost or changed against the
    slot-order push (the sorted columns: three steps round values and sums of
    order 1 a few times, 1e-6 in FP32; particles lie 0.01 apart)."""
    n, ppc, weight = (8, 8, 64), 4, 0.01 / 4
    cells = np.stack(np.meshgrid(*[np.arange(2, m - 2) for m in n], indexing="ij"), -1).reshape(-1, 1, 3)
    xyz = 2 + np.broadcast_to(cells + 0.5, (len(cells), ppc, 3)) + np.linspace(-0.04, 0.04, ppc)[:, None]
    z = np.broadcast_to(cells[..., 2] % 32, xyz.shape[:2])
    xyz[..., 2] += 0.4 * np.sign(16 - z)  # about to leave
    v = np.zeros(xyz.shape)
    v[..., 2] = np.where(z < 16, 0.7, np.where(z > 16, -0.7, 0.0))  # towards the group's 17th cell
    rows = np.concatenate([xyz, v, np.full(xyz.shape[:2] + (1,), weight)], -1).reshape(-1, 7)
    cfg = dict(precision=precision, diag_every_step=0, sort_interval=1, add_interval=1000)

    def load(capacity, slot_order=0):
        P = Pic3D(PicConfig.normalized(*n, 4, capacity=capacity, slot_order=slot_order, **cfg))
        P.init_grid()
        for s in (ION, ELECTRON):
            P.set_particles(s, rows)
        return P

    low, high = len(rows), 200000  # high: a capacity that holds the layout
    while low < high:
        mid = (low + high) // 2
        with load(mid) as P:
            try:
                P.sorting()
                high = mid
            except PicError:
                low = mid + 1
    with load(high) as T, load(high, 1) as S:
        T.sorting()
        for _ in range(3):
            T.step(1)
            S.step(1)
            for s in (ION, ELECTRON):
                a, b = (np.sort(P.particles(s), axis=0) for P in (T, S))
                assert len(a) == len(b) == len(rows)
                assert np.abs(a - b).max() < 1e-4
