"""The bench line's roofline fraction: of the DRAM traffic a step moves where
that is known, so that it is at most 1 however much of the state a step leaves
out; of the algorithmic bytes, named as such, elsewhere."""
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))


def test_fraction_is_of_the_traffic_where_it_is_known():
    import bench
    pc = bench.step_traffic(bench.DEFAULT_WORKLOAD)
    cells, sec, peak = 4096 * 4096, 1.54e-3, 6793.0  # a step of mostly dry canvas: 660 B a cell would be 1.06 of the peak
    r = bench.step_roofline(cells, sec, 660, pc, peak, "measured", "step")
    assert r["basis"] == "measured DRAM traffic"
    assert abs(r["frac"] - pc * cells / sec / 1e9 / peak) < 1e-12 and r["frac"] < 1.0
    assert r["alg_gbs"] > peak
    r = bench.step_roofline(cells, 2e-3, 392, None, peak, "measured", "step")
    assert r["basis"] == "algorithmic bytes" and r["achieved"] == r["alg_gbs"]
