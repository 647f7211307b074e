"""The tracker's iteration schedule: sessions move through their levels and
iterations independently inside one launch.  Levels without iterations, one
level only, images smaller than a range and images of many ranges track as the
oracle does on the same inputs; batches of more sessions than a warp has lanes
give each session what it has alone."""
import numpy as np
import pytest

import helpers
import vs_scanner as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,levels,iters", [(97, 75, 3, (10, 5, 4)), (160, 120, 3, (4, 0, 3)),
                                              (160, 120, 2, (6, 4, 0)), (130, 100, 1, (8, 0, 0)),
                                              (320, 240, 3, (0, 5, 4)), (1280, 960, 3, (3, 2, 2))])
def test_levels_and_iterations_follow_the_configuration(gpu, w, h, levels, iters):
    case = helpers.make_case(width=w, height=h, dim=96, size=1.0, frames=3, seed=12, iters=iters, cos_normal=0.94)
    cfg = case["cfg"]
    cfg.levels = levels
    helpers.reanchored_track_check(case["depth"], cfg, 3, expect_tracked=False)
    with V.Session(cfg) as s:
        for k in range(2):
            s.scan_frame_host(case["depth"][k])
        assert s.pose()[2][1] <= sum(iters[:levels])


def test_no_iteration_at_all_keeps_the_pose(gpu):
    case = helpers.make_case(width=64, height=48, dim=32, size=1.0, frames=2, seed=12, iters=(0, 0, 0))
    with V.Session(case["cfg"]) as s:
        for k in range(2):
            T, tracked = s.scan_frame_host(case["depth"][k])
            assert tracked and np.array_equal(T, np.eye(4, dtype=np.float32))
            assert s.pose()[2][3] == k + 1


def test_forty_sessions_each_as_alone(gpu):
    sizes = [(64, 48), (97, 75), (160, 120)]
    iters = [(10, 5, 4), (3, 0, 2), (5, 5, 0)]
    cases = [helpers.make_case(width=sizes[i % 3][0], height=sizes[i % 3][1], dim=32, size=1.0, frames=3, seed=20 + i,
                               iters=iters[(i // 3) % 3], cos_normal=0.94) for i in range(40)]
    alone = []
    for c in cases:
        with V.Session(c["cfg"]) as s:
            for k in range(3):
                s.scan_frame_host(c["depth"][k])
            alone.append(s.pose())
    sessions = [V.Session(c["cfg"]) for c in cases]
    try:
        with V.Batch() as b:
            for k in range(3):
                b.step_host(sessions, [c["depth"][k] for c in cases])
            for s, ref in zip(sessions, alone):
                got = s.pose()
                assert np.array_equal(got[1], ref[1]) and np.array_equal(got[2], ref[2])
    finally:
        for s in sessions:
            s.close()


@pytest.mark.parametrize("angle", [0.0, 0.02, 0.3])
@pytest.mark.parametrize("mode", [V.VS_REDUCE_FP32, V.VS_REDUCE_KAHAN, V.VS_REDUCE_FP64])
def test_one_iteration_solves_and_applies_its_own_system(gpu, angle, mode):
    """x solves the recorded normal equations and the pose becomes
    exp(x) init T_gc, for steps on both sides of the exponential's series
    range (0.1 rad).  x is recorded in float (relative 2^-24) from an FP64
    solve (relative error below 1e-15 times the condition number)."""
    import torch
    from scipy.linalg import expm

    case = helpers.make_case(width=160, height=120, dim=96, size=1.0, frames=2, seed=9, iters=(1, 0, 0), th_icp=0.25,
                             reduce_mode=mode)
    c, s_ = np.cos(angle), np.sin(angle)
    init = np.eye(4, dtype=np.float32)
    init[:2, :2] = [[c, -s_], [s_, c]]
    with V.Session(case["cfg"]) as s:
        s.scan_frame_host(case["depth"][0])
        T0 = s.pose()[1]
        s.stage_filter(torch.from_numpy(case["depth"][1].view(np.int16)).cuda().data_ptr())
        s.sync()
        assert s.tp_track_pose(torch.from_numpy(init).cuda().data_ptr())
        T1, (sums, x) = s.pose()[1], s.icp_system()
    A = np.zeros((6, 6))
    A[np.triu_indices(6)] = sums[:21]
    A = A + np.triu(A, 1).T
    ref = np.linalg.solve(A, sums[21:27])
    tol = (2.0 ** -24 + 1e-15 * np.linalg.cond(A)) * 2.0
    assert np.linalg.norm(x - ref) <= tol * np.linalg.norm(ref)
    w, v = ref[:3], ref[3:]
    xi = np.zeros((4, 4))
    xi[:3, :3] = [[0, -w[2], w[1]], [w[2], 0, -w[0]], [-w[1], w[0], 0]]
    xi[:3, 3] = v
    want = expm(xi) @ init.astype(np.float64) @ T0
    assert np.abs(T1 - want).max() <= 1e-12 * np.linalg.cond(A)
    print(angle, mode, np.linalg.norm(w), np.linalg.cond(A))
