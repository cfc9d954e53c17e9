"""The FP32 push and drift loops called by themselves over the tiled layout
keep what slot order has in precision: correctly rounded square roots and
divisions, and FP32 sums however uneven the tile's cells are."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION, Pic3D, PicConfig
from util import NE, NI, match_rows

pytestmark = pytest.mark.gpu

N = (8, 8, 40)


def context(slot_order=0, **kw):
    P = Pic3D(PicConfig.normalized(*N, 4, precision=32, diag_every_step=0, sort_interval=1000, add_interval=1000,
                                   slot_order=slot_order, capacity=200000, **kw))
    P.init_grid()
    return P


def test_velocities_are_as_exact_as_in_slot_order():
    """No fields: a push leaves every velocity as it is, but for the roundings
    of its square roots and divisions. The layout's and slot order's are the
    same operations on the same velocities; contracted differently they may
    differ in single cases, not in the mean of 60000 (half a per cent of the
    rms error; the fast square root and division add two)."""
    rng = np.random.default_rng(1)
    xyz = 2 + rng.random((20000, 3)) * np.array(N)
    v = rng.normal(0, 0.2, xyz.shape).astype(np.float32).astype(np.float64)
    rows = np.column_stack([xyz, v, np.full(len(xyz), 0.01 / 4)])
    rms = []
    for slot_order in (0, 1):
        with context(slot_order, coil_i=0.0, imf_x=0.0, imf_y=0.0, imf_z=0.0, v_drift=0.0, absorb_grid2=0) as P:
            P.set_particles(ION, rows)
            P.set_particles(ELECTRON, rows)
            P.sorting()
            P.renew_grid()
            P.push_deposit_j()
            after = rows.copy()
            after[:, :3] += 0.5 * P.cfg.dt * v
            mine, ref = match_rows(P.particles(ION), after)
            rms.append(np.sqrt(((mine[:, 3:6] - ref[:, 3:6]) ** 2).sum() / (ref[:, 3:6] ** 2).sum()))
    assert rms[0] <= 1.005 * rms[1], rms


def test_sparse_cells_beside_a_crowd():
    """Single resting particles in the tile of a cell that holds 20000. Offsets
    are multiples of 2^-8, so each of a particle's eight weights has at most
    24 bits and is rounded when it is scaled by the particle's own weight, and
    once more in each product: 4 x 2^-24 of the node's density."""
    rng = np.random.default_rng(2)
    crowd = np.array([2, 2, 2]) + (rng.integers(1, 256, (20000, 3))) / 256
    cells = np.array([[3, 5, k] for k in range(6, 32, 4)])
    single = cells + rng.integers(1, 256, cells.shape) / 256
    xyz = np.concatenate([crowd, single])
    rows = np.column_stack([xyz, np.zeros_like(xyz), np.full(len(xyz), 0.01 / 4)])
    with context() as P:
        for s in (ION, ELECTRON):
            P.set_particles(s, rows)
        P.sorting()
        P.renew_grid()
        P.drift_deposit_n()
        g = P.grid()
    for x in single:
        base = np.floor(x - 0.5).astype(int)
        f = x - 0.5 - base
        for d in np.ndindex(2, 2, 2):
            w = np.prod(np.where(d, f, 1 - f)) * float(np.float32(0.01 / 4))
            for q in (NI, NE):
                assert abs(g[tuple(base + d) + (q,)] - w) <= 4 * 2.0 ** -24 * w
