"""Which particles thrust_f counts as inside its central box (0.2 N dx, 0.8 N dx):
positions on the faces, one rounding to either side of them, and elsewhere, in
the tiled layout and in slot order."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION, Pic3D, PicConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("dx", [1.0, 1.5, 0.1])
@pytest.mark.parametrize("n", [(5, 5, 5), (7, 12, 33), (20, 10, 64), (13, 9, 70)])
def test_box_faces(n, dx, precision):
    rng = np.random.default_rng(n[2])
    pos = (2 + rng.random((4000, 3)) * np.array(n)) * dx
    for a in range(3):  # a quarter of the particles sits at a face of each axis
        f = np.array([0.2, 0.8])[rng.integers(0, 2, 1000)] * n[a] * dx
        x = [f, np.nextafter(f, 0), np.nextafter(f, 1e9), f * (1 - 2.0 ** -24), f * (1 + 2.0 ** -24)]
        pos[1000 * a:1000 * (a + 1), a] = np.choose(rng.integers(0, 5, 1000), x)
    pos = pos[((pos >= 2 * dx) & (pos < (np.array(n) + 2) * dx)).all(1)]
    rows = np.column_stack([pos, np.full(pos.shape, 0.01), np.full(len(pos), 0.01 / 4)])
    inside = []
    for slot_order in (0, 1):
        cfg = PicConfig.normalized(*n, 4, precision=precision, slot_order=slot_order, capacity=200000, dx=dx)
        with Pic3D(cfg) as P:
            P.init_grid()
            for s in (ION, ELECTRON):
                P.set_particles(s, rows)
            P.sorting()
            x = P.particles(ION)[:, :3]  # as stored, which is what the sums compare
            want = np.ones(len(x), bool)
            for a in range(3):
                size = float(n[a]) * dx
                want &= (x[:, a] > size * 0.2) & (x[:, a] < size * 0.8)
            _, E = P.thrust_f()
            v2 = float(np.sum(P.particles(ION)[0, 3:6] ** 2))
            for q, m in ((2, cfg.mi), (3, cfg.me)):
                count = E[q] / (0.5 * m * (0.01 / 4) * dx ** 3 * v2)
                assert abs(count - want.sum()) < 1e-6
            inside.append(want.sum())
    assert inside[0] == inside[1] and inside[0] > 0
