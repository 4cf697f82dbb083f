"""Figures that bench.py forms from counters follow from what those count."""
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))


def test_fuzzy_set_line_claims_no_exponentials():
    """smooth_knn_steps counts bisection steps, most of which evaluate nothing."""
    import bench
    line = bench.fuzzy_set_line(2.0, 1000, 15, 20_000, 27_000, 6800.0)
    assert not [key for key in line if "exp" in key]
    assert line["mean_bisection_steps_per_row"] == 27.0 and line["smooth_knn_steps"] == 27_000
    assert line["hbm_bytes"] == 8 * 1000 * 15 + 8 * 1001 + 8 * 20_000 + 8 * 1000
    assert line["achieved_gbs"] == round(line["hbm_bytes"] / 2e-3 / 1e9, 1)
