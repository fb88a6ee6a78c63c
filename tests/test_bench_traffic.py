"""roofline.traffic_source says that the autotuned plan's figure stands in for its launches."""
from __future__ import annotations

import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_the_autotuned_plans_traffic_is_called_a_stand_in():
    sys.path.insert(0, str(ROOT))
    import bench

    assert "stand-in" in bench.traffic_source("auto")
    assert "stand-in" not in bench.traffic_source("cholesky")
    # the rows labelled auto are single launches: their comment says so too
    text = (ROOT / "profiles" / "dram_traffic.txt").read_text()
    assert "one launch over a whole side" in text
