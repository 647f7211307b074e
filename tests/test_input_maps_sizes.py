"""Input vertex / normal maps and the tracker's pixel list over the sizes where
their passes change form: one word per row, partial words, the sweep's one and
two words per lane (1024 pixels), masks that fit shared memory and masks that
do not (16384 words)."""
import numpy as np
import pytest

import helpers
import oracle_py as O
import vs_scanner as V

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("w,h", [(24, 18), (32, 33), (97, 41), (1024, 64), (1025, 70), (1290, 420)])
def test_maps_and_listed_tracking(gpu, w, h):
    c = helpers.make_case(width=w, height=h, dim=64, size=1.2, frames=2, seed=4, cos_normal=float(np.cos(np.radians(20.0))),
                          iters=(3, 2, 0))
    cfg = c["cfg"]
    cfg.levels = 2
    K = O.level_K(O.config_from_vs(cfg))
    with V.Session(cfg) as s:
        for k in range(2):  # the second frame's maps replace the first's
            d = torch.from_numpy(np.ascontiguousarray(c["depth"][k]).view(np.int16)).cuda()
            s.stage_filter(d.data_ptr())
            s.sync()
            for l in range(2):
                m = s.maps(l)
                v, n = O.point_normal_map(m["input_depth"], K[l])
                assert np.array_equal(m["input_vertex"], v), (k, l)
                assert np.array_equal(m["input_normal"], n), (k, l)
    # the first iteration's sums over the list against the oracle's over every
    # pixel: the same pixels count, and FP64 sums of the same float terms
    # differ by their order alone
    cfg.levels, cfg.icp_iters[0], cfg.icp_iters[1], cfg.reduce_mode = 1, 1, 0, V.VS_REDUCE_FP64
    ocfg = O.config_from_vs(cfg)
    with V.Session(cfg) as s:
        s.scan_frame_host(c["depth"][0])
        before = s.maps(0)
        d = torch.from_numpy(np.ascontiguousarray(c["depth"][1]).view(np.int16)).cuda()
        s.stage_filter(d.data_ptr())
        s.tp_track_pose()
        sums, now = s.icp_system()[0], s.maps(0)
    ref = np.asarray(O.icp_sums(ocfg, 0, now["input_depth"], before["model_vertex"], before["model_normal"],
                                np.eye(4, dtype=np.float32), innrm=now["input_normal"]), np.float64)
    print(w, h, sums[27], ref[27] if ref.size > 27 else ref)
    assert sums[27] == ref[27]
    assert np.abs(sums - ref).max() <= 1e-10 * np.abs(ref).max()  # w h 2^-53 of the sums of magnitudes, at most
