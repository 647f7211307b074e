"""The counters that one integration hands to the next: after any number of
integrations, a lost frame, a snapshot's load and a reset, an integration lists
the sub-cubes (and counts the voxels) that it lists in a fresh session."""
import numpy as np
import pytest

import helpers
import oracle_py as O
import vs_scanner as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [0, 1, 2, 3])
@pytest.mark.parametrize("event", ["none", "lost", "snapshot", "reset"])
def test_counters_over_events(gpu, tmp_path, before, event):
    import torch

    c = helpers.make_case(width=97, height=75, dim=64, frames=2, seed=6)
    T = [g.astype(np.float32) for g in c["gt"]]
    dev = [[torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (O.depth_to_m(c["depth"][k]), T[k], O.pose_inverse(T[k]))] for k in range(2)]

    def integrate(s, k):
        s.cdtoc_convert_depth_to_tsdf(*[a.data_ptr() for a in dev[k]])
        return np.sort(s.active_bricks()), s.frame_stats()[1]

    expect = []
    for k in range(2):
        with V.Session(c["cfg"]) as f:
            expect.append(integrate(f, k))
    assert not np.array_equal(expect[0][0], expect[1][0])

    s = V.Session(c["cfg"])
    for i in range(before):
        got = integrate(s, i % 2)
        assert np.array_equal(got[0], expect[i % 2][0]) and got[1] == expect[i % 2][1]
    if event == "lost":  # the first frame always counts as tracked; no depth loses the second
        s.scan_frame_host(c["depth"][0])
        _, tracked = s.scan_frame_host(np.zeros_like(c["depth"][0]))
        assert not tracked and s.active_bricks().size == 0 and s.frame_stats()[1] == 0
    elif event == "snapshot":
        s.save(str(tmp_path / "s.vs"))
        s.close()
        s = V.Session.load(str(tmp_path / "s.vs"))
    elif event == "reset":
        s.reset()
    for i in range(3):
        got = integrate(s, (i + 1) % 2)
        assert np.array_equal(got[0], expect[(i + 1) % 2][0]) and got[1] == expect[(i + 1) % 2][1], i
    s.close()
