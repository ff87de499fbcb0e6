"""bench.py's roofline: what the timed kernel moves, or nothing; the bytes of
the reference's walk stand under a name of their own."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
import bench


@pytest.mark.parametrize("workload", ["instanced", "large"])
@pytest.mark.parametrize("captured", [False, True])
def test_reference_work_is_not_the_kernels_rate(monkeypatch, workload, captured):
    fig = {"dram_bytes_per_visit": 2.0, "l1tex_bytes_per_visit": 40.0} if captured else None
    monkeypatch.setattr(bench, "profile_figures", lambda name: (fig, "here"))
    monkeypatch.setattr(bench, "l1_peak_gbs", lambda clocks, device=0: 40_000.0)
    monkeypatch.setattr(bench, "measured_peaks", lambda: (6_800.0, "measured"))
    out = bench.roofline_block(1e12, 0.1, workload, None, "p", 0, 1e10)
    assert out["reference_work"]["achieved"] == 1e4 and "reference" in out["reference_work"]["note"]
    if not captured:
        assert out["achieved"] is None and out["frac"] is None
    elif workload == "large":
        assert out["achieved"] == pytest.approx(200.0) and out["frac"] == pytest.approx(200.0 / 6_800.0)
    else:
        assert out["achieved"] == pytest.approx(4_000.0) and out["frac"] == pytest.approx(0.1)
