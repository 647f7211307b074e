"""The filter of uint16 frames under every depth scale a session accepts: scaled
depth that is negative, infinite or not a number comes out of the filter as the
oracle's arithmetic gives it, as from a float map."""
import numpy as np
import pytest
import torch

import oracle_py as O
import vs_scanner as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.001, -0.001, 0.0, 1e-42, 1e30, 5e33, 1e34, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("w,h", [(40, 24), (33, 17)])
def test_filter_of_scaled_frames(gpu, scale, w, h):
    r = np.random.default_rng(5)
    mm = (20000 + 40000 * r.random((h, w))).astype(np.uint16)
    mm[r.random((h, w)) < 0.02] = 0
    mm[h // 2:h // 2 + 2, :3] = 0
    dev = torch.from_numpy(mm.view(np.int16)).cuda()
    with np.errstate(all="ignore"), V.Session(V.default_config(w, h, dim=(8, 8, 8), levels=1, depth_scale=scale)) as s:
        s.stage_filter(dev.data_ptr())
        s.sync()
        raw, got = s.input_raw(), s.maps(0)["input_depth"]
        ref_raw = mm.astype(np.float32) * np.float32(scale)
        ref = O.bilateral(ref_raw)
    assert np.array_equal(raw, ref_raw, equal_nan=True)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isinf(got), np.isinf(ref))
    assert np.array_equal(got == 0, ref == 0)
    ok = np.isfinite(ref)
    assert (np.abs(got[ok] - ref[ok]) <= 1e-5 * np.maximum(1.0, np.abs(ref[ok]))).all()
