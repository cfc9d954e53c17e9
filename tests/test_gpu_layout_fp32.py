"""The FP32 fused push over crowded and ragged layouts against slot order: the
packed home sums, the window gather and the fixed-point densities. Two steps'
velocities differ by the roundings of the square roots and divisions (2e-7
each, a few of them: 2e-6), their sums by as much, so 1e-5, as for the push and
drift called by themselves; densities are resolved to 2^-32 of the tile's slots
(at most 40 rows of 32 lanes in 8 groups here: 2^-18 of one
particle's weight)."""
import numpy as np
import pytest

from plasmasim_b200 import ELECTRON, ION
from test_gpu_layout import context, crowd
from util import rel_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(8, 8, 8), (5, 7, 31), (6, 5, 33), (9, 6, 64)])
@pytest.mark.parametrize("speed", [0.1, 0.9])
def test_fused_push_over_the_layout(n, speed):
    rng = np.random.default_rng(sum(n) + int(10 * speed))
    rows = [crowd(n, rng, speed) for _ in range(2)]
    with context(n, 32, 0) as T, context(n, 32, 1) as S:
        for s in (ION, ELECTRON):
            T.set_particles(s, rows[s])
            S.set_particles(s, rows[s])
        T.sorting()
        T.step(2)
        S.step(2)
        g, h = T.grid(), S.grid()
        assert np.isfinite(g).all()
        for q in range(18):
            assert rel_norm(g[..., q], h[..., q]) < 1e-5 or np.abs(g[..., q] - h[..., q]).max() < 1e-15
        assert T.status()[0] == S.status()[0] == 0
