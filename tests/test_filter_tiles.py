"""The bilateral filter over sizes around its 32 x 16 tiles and its two rows per
thread, and on values that sums must not hide: negative depth and -infinity are
holes, NaN and +infinity come out as the oracle's arithmetic gives them."""
import numpy as np
import pytest

import oracle_py as O
import vs_scanner as V

pytestmark = pytest.mark.gpu


def depth_map(w, h, seed, special):
    r = np.random.default_rng(seed)
    d = (1.0 + 0.2 * r.random((h, w)) + (r.random((h, w)) > 0.7)).astype(np.float32)
    d[r.random((h, w)) < 0.02] = 0.0
    d[h // 2:h // 2 + 2, :3] = 0.0  # a 2x2 hole: a tap of 0
    if special:
        for v in (-0.5, -np.inf, np.inf, np.nan, 1e30, -3.0):
            d[r.integers(0, h), r.integers(0, w)] = v
    return d


@pytest.mark.parametrize("w,h", [(8, 8), (31, 15), (32, 16), (33, 17), (64, 33), (65, 50), (200, 9)])
@pytest.mark.parametrize("special", [False, True])
def test_filter_over_tile_edges(gpu, w, h, special):
    d = depth_map(w, h, 7, special)
    with np.errstate(all="ignore"), V.Session(V.default_config(w, h, dim=(8, 8, 8), levels=1)) as s:
        got, ref = s.bfd_bilateral_filter_depth_host(d), O.bilateral(d)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
    assert np.array_equal(got == 0, ref == 0)
    ok = np.isfinite(ref)
    assert (np.abs(got[ok] - ref[ok]) <= 1e-5 * np.maximum(1.0, np.abs(ref[ok]))).all()
