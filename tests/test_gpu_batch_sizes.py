"""A 2D run gives the same result whatever batch it is in: small batches take
smaller items in the field updates and the sine transforms (32 x 32 output
tiles instead of 64 x 64), at sides that neither divides."""
import numpy as np
import pytest

from plasmasim_b200 import Pic2DBatch, Pic2DConfig
from util import rel_norm

pytestmark = pytest.mark.gpu


def config(nx, nz, r, np_=2):
    return Pic2DConfig(nx=nx, nz=nz, np=np_, add_interval=3, absorb_grid=8, absorb_grid2=4, absorb_grid3=8,
                       seed_p=100 + r, seed_v=200 + r, sort_interval=2)


@pytest.mark.parametrize("side", [(64, 64), (66, 130), (100, 76), (97, 33)])
def test_run_does_not_depend_on_its_batch(side):
    crowd = [config(128, 128, r, 1) for r in range(1, 80)]  # 316 tiles of 64 x 64, 10112 rows
    with Pic2DBatch([config(*side, 0)], precision=64) as A, \
            Pic2DBatch([config(*side, 0)] + crowd, precision=64) as B:
        for b in (A, B):
            b.init()
            b.step(5)
        g, h = A.grid(0), B.grid(0)
        # the products' terms and the particles' sums in another order
        for q in range(18):
            assert rel_norm(g[..., q], h[..., q]) < 1e-11 or np.abs(g[..., q] - h[..., q]).max() < 1e-13
        t, u = A.thrust()[0], B.thrust()[0]
        assert np.abs(t - u).max() <= 1e-9 * np.abs(u).max()
        assert [A.count(0, s) for s in (0, 1)] == [B.count(0, s) for s in (0, 1)]
        assert A.status()[0] == B.status()[0] == 0
