"""Rays that march longer than the 64 turns after which the ray-cast looks for
repetition, and hit: in free space of small TSDF a fine step is one voxel, so a
surface `z` voxels behind the volume's front is some `z` turns away.  Stripes of
surfaces on both sides of 64 turns stand beside stripes whose rays repeat."""
import numpy as np
import pytest

import helpers
import oracle_py as O
import vs_scanner as V

DIM = 160
STRIPE = 16                                                      # voxels along x
DEPTHS = (30, 56, 62, 64, 66, 72, 90, 110, 130, 145)             # of the stripes' surfaces


def stripes(repeat_gap):
    """TSDF 0.1 up to each stripe's surface, -0.1 behind it; in every second row
    of 16 voxels along y a slab of `repeat_gap` voxels of weight 0 with exactly
    -1 behind it instead, which sends rays back and forth"""
    t = np.full((DIM, DIM, DIM), 0.1, np.float32)
    w = np.ones((DIM, DIM, DIM), np.uint16)
    for k, z in enumerate(DEPTHS):
        x = slice(k * STRIPE, (k + 1) * STRIPE)
        for y0 in range(0, DIM, 32):
            t[z:, y0:y0 + 16, x] = -0.1
            w[z:z + repeat_gap, y0 + 16:y0 + 32, x] = 0
            t[z:, y0 + 16:y0 + 32, x] = -1.0
    return t.reshape(-1), w.reshape(-1)


def make(tsdf):
    return helpers.make_case(width=160, height=120, dim=DIM, size=1.0, frames=1, seed=1, mu=5.0 / DIM, tsdf_type=tsdf)


def oracle_depth(case, t, w):
    vol = O.Volume(case["ocfg"])
    vol.set(t, w)
    T = np.eye(4, dtype=np.float32)
    return vol.raycast(0, T, T, O.camera_center(T))[0]


def hit_layer(case, depth):
    """voxels between the volume's front and each hit (0: none)"""
    cfg = case["cfg"]
    return np.where(depth > 0, (depth - cfg.origin[2]) / cfg.voxel_size, 0.0)


@pytest.mark.parametrize("gap", [2, 6])
def test_stripes_hold_long_hits_and_repeating_rays(gap):
    case = make(V.VS_TSDF_FP32)
    layer = hit_layer(case, oracle_depth(case, *stripes(gap)))
    print([(z, int((np.abs(layer - z) < 2).sum())) for z in DEPTHS], (layer == 0).sum())
    for lo, hi in ((20, 60), (60, 64), (64, 70), (70, 160)):
        assert ((layer > lo) & (layer <= hi)).sum() > 300, (lo, hi)
    assert (layer == 0).sum() > 2000


@pytest.mark.gpu
@pytest.mark.parametrize("tsdf", [V.VS_TSDF_INT16, V.VS_TSDF_FP16, V.VS_TSDF_FP32])
@pytest.mark.parametrize("gap", [2, 6])
def test_long_rays_hit_beside_repeating_ones(gpu, gap, tsdf):
    """the ray-cast's contract (99.9 % of the hit mask, 1 mm), of which the
    rays that hit after more than 64 turns are more than a twentieth"""
    torch = pytest.importorskip("torch")
    case = make(tsdf)
    t, w = stripes(gap)
    od = oracle_depth(case, t, w)
    assert (hit_layer(case, od) > 70).mean() > 0.05
    with V.Session(case["cfg"]) as s:
        s.set_volume(t, w)
        out = [torch.zeros(od.size * c, dtype=d, device="cuda") for c, d in
               ((1, torch.float32), (3, torch.float32), (3, torch.float32), (1, torch.uint8))]
        e = torch.eye(4, device="cuda")
        torch.cuda.synchronize()
        s.rmi_render_maps_for_icp(0, e.data_ptr(), e.data_ptr(), np.zeros(3, np.float32), (0, 0, -1),
                                  *[o.data_ptr() for o in out])
        gd = out[0].cpu().numpy().reshape(od.shape)
    assert ((gd > 0) == (od > 0)).mean() >= 0.999
    both = (gd > 0) & (od > 0)
    assert (np.abs(gd[both] - od[both]) <= 1e-3).mean() >= 0.999
