"""Rays whose signed fine steps return them to where they were: the reference
repeats them until its iteration cap and reports no hit; the ray-cast ends
them when it sees the repetition.  A slab of weight 0 between free space and
voxels that read exactly -1 sends a ray back and forth for every step length."""
import numpy as np
import pytest

import helpers
import oracle_py as O
import vs_scanner as V


def slabs(case, gap):
    """TSDF 0.5 up to a slab of `gap` voxels of weight 0, -1 behind it (along z)"""
    n = case["cfg"].dim[0]
    t = np.full((n, n, n), 0.5, np.float32)
    w = np.ones((n, n, n), np.uint16)
    z = n // 2
    w[z:z + gap] = 0
    t[z:] = -1.0
    return t.reshape(-1), w.reshape(-1)


def oracle_maps(case, t, w):
    vol = O.Volume(case["ocfg"])
    vol.set(t, w)
    T = np.eye(4, dtype=np.float32)
    return vol.raycast(0, T, T, O.camera_center(T))


@pytest.mark.gpu
@pytest.mark.parametrize("tsdf", [V.VS_TSDF_INT16, V.VS_TSDF_FP16, V.VS_TSDF_FP32])
@pytest.mark.parametrize("voxels,gap", [(3.3, 2), (3.3, 6), (5.0, 3), (5.0, 6), (7.7, 10)])
def test_repeating_rays_report_no_hit(gpu, voxels, gap, tsdf):
    torch = pytest.importorskip("torch")
    case = helpers.make_case(width=64, height=48, dim=64, size=1.0, frames=1, seed=1, mu=voxels / 64.0, tsdf_type=tsdf)
    t, w = slabs(case, gap)
    od, ov, _, _ = oracle_maps(case, t, w)
    with V.Session(case["cfg"]) as s:
        s.set_volume(t, w)
        h, wd = od.shape
        out = [torch.zeros(h * wd * c, dtype=d, device="cuda") for c, d in
               ((1, torch.float32), (3, torch.float32), (3, torch.float32), (1, torch.uint8))]
        e = torch.eye(4, device="cuda")
        torch.cuda.synchronize()
        s.rmi_render_maps_for_icp(0, e.data_ptr(), e.data_ptr(), np.zeros(3, np.float32), (0, 0, -1),
                                  *[o.data_ptr() for o in out])
        gd = out[0].cpu().numpy().reshape(h, wd)
    assert ((gd > 0) == (od > 0)).mean() >= 0.999
    both = (gd > 0) & (od > 0)
    assert (np.abs(gd[both] - od[both]) <= 1e-3).all()
    assert (od == 0).mean() > 0.5  # most rays repeat
