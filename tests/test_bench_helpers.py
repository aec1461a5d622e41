"""The measurement arithmetic of bench.py on the CPU: the non-walk stages' HBM
roofline (algorithmic bytes per particle, cell and group; the reference's
IOCOUNT build accounting) and the log-log interpolation of the fixed-angle
sweep at equal error that the learned form is judged against."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_hbm_roofline_bytes_and_fraction():
    import bench
    n, info, ms = 1 << 20, {"ncells": 250000, "ngroups": 17000, "nlevels": 12}, 0.5
    r = bench.hbm_roofline(n, info, ms)
    want = n * (28 + 24 + 64 + 8 + 16 + 8 + 80) + 250000 * (16 + 72) + 8 * 17000
    assert r["algorithmic_bytes_per_step"] == want
    assert r["achieved"] == pytest.approx(want / (ms * 1e-3) / 1e9)
    assert r["frac"] == pytest.approx(r["achieved"] / r["peak"])
    assert r["reference_build_bytes"] == 32.0 * n * 12
    assert r["bound"] == "hbm" and r["unit"] == "GB/s"


def test_at_equal_interpolates_log_log_inside_the_sweep_only():
    import bench
    sweep = [{"v": 100.0, "e": 1e-4}, {"v": 400.0, "e": 1e-3}, {"v": 200.0, "e": 3e-4}]
    # exact at the points, log-log linear between them
    assert bench.at_equal(sweep, "v", "e", 1e-4) == pytest.approx(100.0)
    assert bench.at_equal(sweep, "v", "e", 1e-3) == pytest.approx(400.0)
    mid = np.sqrt(3e-4 * 1e-3)
    assert bench.at_equal(sweep, "v", "e", mid) == pytest.approx(np.sqrt(200.0 * 400.0))
    # outside the measured range there is no number
    assert bench.at_equal(sweep, "v", "e", 5e-5) is None
    assert bench.at_equal(sweep, "v", "e", 2e-3) is None


def test_workload_names_the_configuration():
    import types
    import bench
    a = types.SimpleNamespace(n=1 << 24, theta=0.6, eps=0.005, nleaf=16, ncrit=64, level_split=5, dt=1.0 / 128,
                              seed=19810614)
    w = bench.workload(a)
    assert "N=16777216" in w and "theta=0.6" in w and "dt=1/128" in w and "FP32" in w


def test_result_line_is_short_and_whole():
    """The line that rank 0 prints carries every figure of the result and stays
    within what a log's tail holds, however long the record."""
    import json
    import bench
    row = {"theta": 0.6, "value": 1.0 / 3, "median_rel_force_err": 2.6e-4 / 3, "what": "x" * 500}
    form = {"value": 1.0 / 3, "ms_per_step": 2.0 / 3, "sweep": [row] * 20, "what": "y" * 2000}
    record = {"metric": bench.METRIC, "value": 245.123456789, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
              "ms_per_step": 68.123456789, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
              "dtype": "f32", "data": "synthetic", "gpu_launches": 760,
              "config": {"workload": "w" * 120, "n_per_gpu": 1 << 24, "parallelism": "replicas x1", "l2": "no flush"},
              "e2e": {"value": 1.0 / 3, "unit": bench.UNIT, "h2d_bytes_per_step": 1 << 29, "d2h_bytes_per_step": 1 << 28},
              "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": []},
              "roofline": {"bound": "fp32", "frac": 1.0 / 3}, "theta_sweep": [row] * 8, "skipped_form": None,
              **{"form%d" % k: dict(form) for k in range(9)}}
    line = bench.result_line(record)
    assert "\n" not in line and len(line) <= bench.MAX_LINE
    got = json.loads(line)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "gpu_launches", "config", "clocks"):
        assert got[k] == record[k], k
    assert got["e2e"]["value"] == pytest.approx(1.0 / 3, rel=1e-6) and got["e2e"]["h2d_bytes_per_step"] == 1 << 29
    assert got["forms"]["form3"]["value"] == pytest.approx(1.0 / 3, rel=1e-6)
    assert len(got["forms"]["theta_sweep"]) == 8
    # forms that do not fit are left out, the result never
    record.update({"f%d" % k: dict(form) for k in range(200)})
    line = bench.result_line(record)
    assert len(line) <= bench.MAX_LINE and json.loads(line)["value"] == record["value"]
