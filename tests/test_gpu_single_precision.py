"""The FP32 push called by itself over the tiled layout keeps what slot order
has in precision: correctly rounded square roots and divisions."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION, Pic3D, PicConfig
from util import match_rows

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
