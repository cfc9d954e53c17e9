"""The capacity of a store: a full sort that does not fit leaves the store as
it was; evenly filled cells need no more slots than rows sized for each group's
fullest cell, a sixteenth and two more."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION, Pic3D, PicConfig, PicError
from util import rel_norm

pytestmark = pytest.mark.gpu


def smallest(fits, low, high):
    """The smallest capacity in (low, high] that `fits` accepts; high does."""
    while low < high:
        mid = (low + high) // 2
        if fits(mid):
            high = mid
        else:
            low = mid + 1
    return high


def refused(call):
    try:
        call()
    except PicError:
        return True
    return False


def canonical(rows):
    rows = np.round(rows, 6)
    return rows[np.lexsort(rows.T[::-1])]


@pytest.mark.parametrize("precision", [32, 64])
def test_a_sort_that_does_not_fit_changes_nothing(precision):
    """Particles that fill the rows reserved for the refill of the low x shell
    and move on along x, in a capacity that the first sort just fills: a later
    sort needs more rows. After it fails, the store holds the particles that it
    held and deposits the same current as slot order (the loop bodies'
    roundings: FP64 1e-11, FP32 1e-5)."""
    n = (9, 8, 32)
    rng = np.random.default_rng(precision)
    rows = []
    for s in (ION, ELECTRON):
        xyz = 2 + rng.random((4000, 3)) * [2, 8, 32]
        v = rng.normal(0, 0.02, xyz.shape) + [0.9, 0, 0]
        rows.append(np.column_stack([xyz, v, np.full(len(xyz), 0.01 / 4)]))

    def load(capacity, slot_order=0):
        P = Pic3D(PicConfig.normalized(*n, 4, precision=precision, capacity=capacity, slot_order=slot_order,
                                       diag_every_step=0, sort_interval=1000, add_interval=1000))
        P.init_grid()
        for s in (ION, ELECTRON):
            P.set_particles(s, rows[s])
        return P

    def fits(capacity):
        with load(capacity) as P:
            return not refused(P.sorting)

    cap = smallest(fits, len(rows[0]), 200000)
    failed = 0
    with load(cap) as T, load(200000, 1) as S:
        T.sorting()
        for body in range(24):
            for P in (T, S):
                P.renew_grid()
                P.push_deposit_j()
                P.drift_deposit_n()
                P.sr_particle()
            if body % 4 == 3:  # a species' failure is reported once, the second one's by the next call
                failed += refused(T.sorting) + (T.status()[0] != 0)
        assert failed
        g, h = T.grid(), S.grid()
        tol = 1e-11 if precision == 64 else 1e-5
        for q in range(18):
            assert rel_norm(g[..., q], h[..., q]) < tol or np.abs(g[..., q] - h[..., q]).max() < 1e-15
        for s in (ION, ELECTRON):
            a, b = T.particles(s), S.particles(s)
            assert len(a) == len(b)
            if precision == 64:
                assert rel_norm(canonical(a), canonical(b)) < 1e-6
        assert T.status()[0] == 0


def refill(n, ppc):
    """Particles that a refill puts into each cell: two layers at both ends of
    z, between them at both ends of y, and low x (over the high y layers too)."""
    need = np.zeros(n, dtype=int)
    need[:, :, :2] += ppc
    need[:, :, -2:] += ppc
    need[:, :2, 2:-2] += ppc
    need[:, -2:, 2:-2] += ppc
    need[:2, 2:, 2:-2] += ppc
    return need


def fullest_slots(n, ppc):
    """Slots of groups of 32 cells along z whose rows hold the group's fullest
    cell (its refill with an eighth and four more, where that is larger) and a
    sixteenth and two more, with ppc particles in every cell."""
    need = refill(n, ppc)
    m = np.maximum(ppc, np.where(need > 0, need + need // 8 + 4, 0))
    m = m.reshape(n[0], n[1], -1, 32).max(axis=-1)
    return int(32 * (m + m // 16 + 2).sum())


@pytest.mark.parametrize("ppc", [4, 16, 64])
def test_even_cells_fit_where_the_fullest_cell_does(ppc):
    """A sort of evenly filled cells, and a refill behind the layout, in a
    capacity of fullest_slots and the refill."""
    n = (10, 12, 256)  # most groups without a shell's cells, no lane without a cell
    cap = fullest_slots(n, ppc) + int(refill(n, ppc).sum())
    with Pic3D(PicConfig.normalized(*n, ppc, precision=32, diag_every_step=0, sort_interval=1000, add_interval=1000,
                                    capacity=cap)) as P:
        P.init_grid()
        P.init_particle_flat()
        P.sorting()
        for s in (ION, ELECTRON):  # without the initial load's particle outside the interior
            assert P.particle_count(s) == ppc * np.prod(n)
        P.add_flat()
        P.step(1)
        assert P.status()[0] == 0
