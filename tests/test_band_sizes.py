"""The band distance field over brick grids around its 32-brick words, its
16-brick reads and its 4-brick stores, against the brute-force transform."""
import numpy as np
import pytest

import vs_scanner as V
from test_band import chebyshev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [(1, 1, 1), (3, 5, 2), (4, 1, 9), (16, 3, 5), (20, 7, 4), (31, 9, 3), (32, 2, 17),
                                (33, 10, 8), (48, 5, 6), (64, 20, 3), (65, 4, 4), (128, 3, 2), (1, 128, 3), (2, 3, 128)])
@pytest.mark.parametrize("flagged", [1, 4])
def test_band_distances_over_grids(gpu, nb, flagged):
    rng = np.random.default_rng(sum(nb) + flagged)
    dim = tuple(8 * n for n in nb)
    want = np.zeros(nb[::-1], np.uint8)
    n = dim[0] * dim[1] * dim[2]
    t, w = np.ones(n, np.float32), np.zeros(n, np.uint16)
    for _ in range(flagged):
        x, y, z = (int(rng.integers(0, d)) for d in dim)
        t[(z * dim[1] + y) * dim[0] + x], w[(z * dim[1] + y) * dim[0] + x] = 0.25, 3
        want[z // 8, y // 8, x // 8] = 1
    with V.Session(V.default_config(32, 24, dim=dim, levels=1)) as s:
        s.set_volume(t, w)
        s.stage_raycast()
        s.sync()
        band, dist = s.band()
    assert np.array_equal(band, want)
    assert np.array_equal(dist, chebyshev(want))
