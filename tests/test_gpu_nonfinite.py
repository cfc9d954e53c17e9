"""What a slot without a particle, or a particle that is not in its lane's home
cell, holds does not reach the sums of the tiled push: removed particles with
NaN and infinite velocities, and live ones that Boris or the domain's end takes
away, against the slot-order push. Tolerances as for the other comparisons of
the two: FP64 1e-11, FP32 1e-5 (a step's square roots and divisions round to
2e-7 each, a few of them)."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION, Pic3D, PicConfig
from util import JEZ, JIX, rel_norm

pytestmark = pytest.mark.gpu

N = (6, 7, 40)
BAD = [np.nan, np.inf, -np.inf]


def contexts(precision, **kw):
    P = []
    for slot_order in (0, 1):
        P.append(Pic3D(PicConfig.normalized(*N, 4, precision=precision, diag_every_step=0, sort_interval=1000,
                                            add_interval=1000, slot_order=slot_order, capacity=100000, **kw)))
        P[-1].init_grid()
    return P


def background(rng, n=3000):
    xyz = 2 + rng.random((n, 3)) * np.array(N)
    return np.column_stack([xyz, rng.normal(0, 0.05, xyz.shape), np.full(n, 0.01 / 4)])


def spoil(rows, rng, where):
    """A copy of `rows` whose rows `where` have a NaN or infinite velocity component each."""
    rows = rows.copy()
    for r in np.flatnonzero(where):
        rows[r, 3 + rng.integers(3)] = BAD[rng.integers(3)]
    return rows


def compare(P, precision, planes=range(18)):
    tol = 1e-11 if precision == 64 else 1e-5
    g, h = P[0].grid(), P[1].grid()
    for q in planes:
        assert np.isfinite(h[..., q]).all() and np.isfinite(g[..., q]).all()
        assert rel_norm(g[..., q], h[..., q]) < tol or np.abs(g[..., q] - h[..., q]).max() < 1e-15


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("call", ["push_deposit_j", "step"])
def test_removed_particles_leave_nothing(call, precision):
    """Particles of a refill shell (z cells 2 and 3), every second one with a
    velocity that is not finite, removed by the refill after a sort."""
    rng = np.random.default_rng(precision)
    P = contexts(precision)
    for s in (ION, ELECTRON):
        rows = background(rng)
        rows = spoil(rows, rng, (rows[:, 2] < 4) & (np.arange(len(rows)) % 2 == 0))
        assert not np.isfinite(rows).all()
        for p in P:
            p.set_particles(s, rows)
    for p in P:
        p.sorting()
        p.add_flat()
        if call == "step":
            p.step(2)
        else:
            p.renew_grid()
            p.push_deposit_j()
    compare(P, precision)
    for s in (ION, ELECTRON):
        assert P[0].particle_count(s) == P[1].particle_count(s)
    (ra, ca), (rb, cb) = P[0].status(), P[1].status()
    assert ra == rb == 0 and np.array_equal(ca, cb)
    for p in P:
        p.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_particles_that_leave_at_infinite_speed(precision):
    """Ballistic particles (the outer 5 cells) of infinite velocity along x
    leave the domain without a deposit; their lanes' sums stay what they are."""
    rng = np.random.default_rng(3 * precision)
    P = contexts(precision, absorb_grid2=5)
    for s in (ION, ELECTRON):
        rows = background(rng)
        rows[::9, 3] = np.inf
        for p in P:
            p.set_particles(s, rows)
    for p in P:
        p.sorting()
        p.renew_grid()
        p.push_deposit_j()
    compare(P, precision)
    for p in P:
        p.close()


@pytest.mark.parametrize("precision", [32, 64])
def test_a_stranger_spoils_its_own_cell_alone(precision):
    """A cell of 300 particles, every tenth with a velocity that is not finite,
    most of them in other cells' lanes: J is not finite at the nodes that this
    cell's particles reach, and nowhere else."""
    rng = np.random.default_rng(5 * precision)
    cell = np.array([4, 5, 20])
    P, S = contexts(precision)
    S.close()
    for s in (ION, ELECTRON):
        crowd = background(rng, 300)
        crowd[:, :3] = cell + rng.random((300, 3))
        crowd = spoil(crowd, rng, np.arange(300) % 10 == 0)
        P.set_particles(s, np.concatenate([background(rng, 400), crowd]))
    P.sorting()
    P.renew_grid()
    P.push_deposit_j()
    bad = np.argwhere(~np.isfinite(P.grid()[..., JIX:JEZ + 1]).all(axis=-1))
    assert len(bad) and np.abs(bad - cell).max() <= 1
    P.close()
