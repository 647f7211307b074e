"""Registration into outputs of odd sizes at unaligned offsets, with many depth
pixels per output pixel, and into memory that overlaps the input: the oracle's
image bit for bit, and nothing written beside it."""
import numpy as np
import pytest

import oracle_py as O
import vs_scanner as V

pytestmark = pytest.mark.gpu

W, H = 97, 61
KD = np.array([90.0, 90.0, 48.0, 30.0], np.float32)


@pytest.mark.parametrize("wr,hr", [(1, 1), (3, 2), (7, 5), (33, 17), (97, 61), (131, 64)])
@pytest.mark.parametrize("offset", [0, 1, 3, 7])
@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("mm", [False, True])
def test_register_outputs(gpu, wr, hr, offset, overlap, mm):
    import torch

    depth = np.random.default_rng(3).integers(0, 65536, (H, W)).astype(np.uint16)
    depth[::5] = 0
    depth[0, :4] = (1, 2, 65534, 65535)
    Kr = np.array([90.0 * wr / W, 90.0 * hr / H, (wr - 1) / 2, (hr - 1) / 2], np.float32)
    T = np.eye(4, dtype=np.float32)
    T[0, 3] = -0.05
    ref = O.warp_depth(O.depth_to_m(depth), KD, T, Kr, wr, hr)
    din = torch.from_numpy(depth.view(np.int16) if mm else O.depth_to_m(depth)).cuda().reshape(-1)
    n, room = wr * hr, max(W * H, wr * hr) + 64
    buf = torch.full((room,), -7, dtype=din.dtype, device="cuda")
    if overlap:
        buf[:W * H] = din
        din = buf
    before = buf.clone()
    out = buf[offset:offset + n]
    V.warp_depth_to_color(din.data_ptr(), W, H, KD, T, Kr, wr, hr, out.data_ptr(), mm_scale=0.001 if mm else None)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    got = O.depth_to_m(got.view(np.uint16)) if mm else got
    assert np.array_equal(got.reshape(hr, wr), ref) and (n == 1 or (ref > 0).any())
    assert torch.equal(buf[:offset], before[:offset]) and torch.equal(buf[offset + n:], before[offset + n:])
