"""Integration over brick counts from a few to more than the kernel's warps (a
brick's update runs in 1, 2 or 4 parts), ragged images and every storage: the
sub-cubes listed, the weights and the band flags exactly, values within one
int16 step.  The start volume is one step below 1 everywhere, so half-precision
free space rounds back to 1 and bricks lose their band flag."""
import numpy as np
import pytest

import helpers
import oracle_py as O
import vs_scanner as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,dim,mu", [(80, 61, 64, 0.03), (97, 75, 128, 0.03), (203, 149, 256, 0.05),
                                         (203, 149, 256, 0.15)])
@pytest.mark.parametrize("tsdf_type", [V.VS_TSDF_INT16, V.VS_TSDF_FP16, V.VS_TSDF_FP32])
@pytest.mark.parametrize("colour", [False, True])
def test_integrate_parts(gpu, w, h, dim, mu, tsdf_type, colour):
    import torch

    c = helpers.make_case(width=w, height=h, dim=dim, frames=2, seed=5, mu=mu, tsdf_type=tsdf_type)
    cfg, n = c["cfg"], dim ** 3
    cfg.color = 1 if colour else 0
    rgb = np.random.default_rng(1).integers(1, 255, (3, h, w), dtype=np.uint8)
    vol = O.Volume(O.config_from_vs(cfg))
    below = {V.VS_TSDF_FP16: 1 - 2.0 ** -11, V.VS_TSDF_INT16: 32766 / 32767, V.VS_TSDF_FP32: 1 - 2.0 ** -24}
    t0 = np.full(n, below[tsdf_type], np.float32)
    w0 = np.ones(n, np.uint16)
    with V.Session(cfg) as s, V.Session(cfg) as ref:
        s.set_volume(t0, w0)
        vol.set(t0, w0)
        for k in range(2):
            raw, Tgc = O.depth_to_m(c["depth"][k]), c["gt"][k].astype(np.float32)
            Tcg = O.pose_inverse(Tgc)
            d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (raw, Tgc, Tcg, rgb)]
            torch.cuda.synchronize()
            if colour:
                vol.integrate_color(raw, rgb, Tgc, Tcg)
                s.cdtocc_convert_depth_to_tsdf_color(d[0].data_ptr(), d[3].data_ptr(), d[1].data_ptr(), d[2].data_ptr())
            else:
                vol.integrate(raw, Tgc, Tcg)
                s.cdtoc_convert_depth_to_tsdf(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr())
            assert np.array_equal(np.sort(s.active_bricks()), np.nonzero(vol.flags())[0].astype(np.uint32))
        t, wgt = s.volume()
        ot, ow = vol.get()
        assert np.array_equal(wgt, ow) and (ow > 1).sum() > 1000
        if colour:
            assert np.array_equal(s.color_volume(), vol.get_color())
        m = ow > 1
        if tsdf_type == V.VS_TSDF_INT16:
            assert np.max(np.abs(helpers.q16(t[m]) - helpers.q16(ot[m]))) <= 1
        else:
            helpers.assert_tsdf_within_one_step(t[m], ot[m])
        ref.set_volume(t, wgt)  # recomputes the flags from the voxels
        assert np.array_equal(s.band()[0], ref.band()[0])
        assert tsdf_type != V.VS_TSDF_FP16 or not s.band()[0].all()
