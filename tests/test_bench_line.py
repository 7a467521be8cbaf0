"""What the benchmark prints: one short line, whole records beside it."""
from __future__ import annotations

import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))


def test_one_short_line(capsys):
    import bench
    sub = {"metric": "m" * 40, "value": 1.23456789e12, "e2e": {"value": 9.87654321e9},
           "config": {"x": "y" * 2500}, "cpu_baseline": {"parity": {"exact": True, "rows": 3}}}
    line = {"metric": "gapblock score_matrix pairs/s", "value": 2.83123456789e11, "ms_per_step": 0.0353201,
            "gpu_launches": 20, "clocks": {"reasons": []},
            "workloads": {**{n: dict(sub) for n in bench.SUITE[:-1]}, "learned": {"error": "x" * 500}},
            "int_peaks": {"lop3": {"all_sms_lane_ops_per_s": 1.0}}}
    bench.emit(line)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) < 2800
    got = json.loads(out)
    assert got["value"] == 2.83123e11 and got["gpu_launches"] == 20
    assert got["workloads"]["sparse"] == {"value": 1.23457e12, "e2e": 9.87654e9, "exact": True}
    whole = [json.loads(t) for t in err.splitlines()]
    assert [t.get("workload") for t in whole] == bench.SUITE + [None]
    assert whole[0]["config"] == sub["config"] and "int_peaks" in whole[-1]


def test_the_reference_arm_times_only_the_reference(capsys, monkeypatch):
    import bench
    import oracle
    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    assert bench.main(["--impl", "reference"]) == 0
    got = json.loads(capsys.readouterr().out)
    assert got["impl"] == "reference" and got["unavailable"]
