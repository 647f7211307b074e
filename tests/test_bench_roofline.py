"""bench.py's roofline entry of a stage: tracking, which reads listed pixels and
stops when converged, states no bandwidth; the counted stages state theirs."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402
import vs_scanner as V  # noqa: E402

STAGES = ("filter", "track", "integrate", "raycast")


def test_stage_rooflines():
    cfg = V.default_config(640, 480, dim=(512, 512, 512))
    alg = bench.stage_bytes(cfg, (8867, 2.0e6))
    ms = dict(zip(STAGES, (0.06, 0.18, 0.04, 0.09)))
    for stage in STAGES:
        r = bench.stage_roofline(stage, alg, ms, 6757.9, "measured", 1.0e6)
        assert r["stage"] == stage and r["traffic"] == 1.0e6 and set(r["stages_gbs"]) == set(STAGES) - {"track"}
        if stage == "track":
            assert (r["bound"], r["achieved"], r["frac"]) == ("latency", None, None)
        else:
            assert r["bound"] == "hbm" and r["achieved"] == pytest.approx(alg[stage] / ms[stage] / 1e6)
            assert r["frac"] == pytest.approx(r["achieved"] / 6757.9)
