"""The bilateral filter of a float map around the size where its threads take
two rows instead of one (912 tiles of 32 x 8 on 152 SMs), holes and non-finite
values included."""
import numpy as np
import pytest

import oracle_py as O
import vs_scanner as V
from test_filter_tiles import depth_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(608, 384), (609, 384), (640, 401), (33, 2048), (1201, 333)])
@pytest.mark.parametrize("special", [False, True])
def test_filter_one_and_two_rows(gpu, w, h, special):
    d = depth_map(w, h, 11, special)
    with np.errstate(all="ignore"), V.Session(V.default_config(w, h, dim=(8, 8, 8), levels=1)) as s:
        got, ref = s.bfd_bilateral_filter_depth_host(d), O.bilateral(d)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
    assert np.array_equal(got == 0, ref == 0)
    ok = np.isfinite(ref)
    assert (np.abs(got[ok] - ref[ok]) <= 1e-5 * np.maximum(1.0, np.abs(ref[ok]))).all()
