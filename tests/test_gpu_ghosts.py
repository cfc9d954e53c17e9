"""The ghost copies that the field updates make themselves, and the one-pass
fold, against the reference's two passes in numpy (bit for bit), from the
smallest sides on: random fields in every node, ghosts and z ends included."""
import numpy as np
import pytest

from plasmasim_b200 import Pic3D, PicConfig
from util import BX, EX, JIX, NE

pytestmark = pytest.mark.gpu


def wrap(a, nx, ny):
    """sr_b / sr_e at size 1: x planes over every (y, z), then y planes over every (x, z)."""
    a = a.copy()
    a[0:2], a[nx + 2:] = a[nx:nx + 2].copy(), a[2:4].copy()
    a[:, 0:2], a[:, ny + 2:] = a[:, ny:ny + 2].copy(), a[:, 2:4].copy()
    return a


def fold(a, nx, ny):
    a = a.copy()
    a[2:4] += a[nx + 2:]
    a[nx:nx + 2] += a[0:2]
    a[:, 2:4] += a[:, ny + 2:]
    a[:, ny:ny + 2] += a[:, 0:2]
    return a


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [(5, 5, 5), (5, 6, 8), (6, 5, 7), (9, 13, 32), (8, 8, 36)])
def test_updates_write_their_ghosts(n, precision):
    nx, ny, _ = n
    rng = np.random.default_rng(nx * ny)
    dt = np.float32 if precision == 32 else np.float64
    with Pic3D(PicConfig.normalized(*n, 1, precision=precision)) as P:
        P.init_grid()
        g = rng.normal(size=P.shape + (18,)).astype(dt).astype(np.float64)
        for op, first in (("renew_b4_2", BX), ("renew_e4_2", EX)):
            P.set_grid(g)
            getattr(P, op)()
            h = P.grid()
            for q in range(first, first + 3):
                # interior and z ends as the update left them, every other column its image
                assert np.array_equal(h[..., q], wrap(h[..., q], nx, ny))
                assert np.array_equal(h[2:nx + 2, 2:ny + 2, :2, q], g[2:nx + 2, 2:ny + 2, :2, q])
                assert np.array_equal(h[2:nx + 2, 2:ny + 2, -2:, q], g[2:nx + 2, 2:ny + 2, -2:, q])
        P.set_grid(g)
        P.reduce_current()
        h = P.grid()
        for q in range(JIX, NE + 1):
            assert np.array_equal(h[..., q], fold(g[..., q].astype(dt), nx, ny).astype(np.float64))
        assert P.status()[0] == 0
