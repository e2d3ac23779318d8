"""The summary of a windowed sweep's rounds (ccd_b200/trace.py) on a synthetic trace in
the engine's file layout."""
import numpy as np

from ccd_b200 import trace


def test_rounds_summary(tmp_path):
    t = np.zeros(8, trace.ROUND)
    for i in range(6):
        t[i] = (1000 * i + 1, 1000 * i + 601, 1000 * i + (801 if i % 2 else 701), 5 * (i % 3), 10, 5, i % 2, 0)
    t[5]["alone"], t[5]["flying"], t[5]["taken"] = 1, 1, 1
    path = tmp_path / "r.bin"
    t.tofile(path)
    out = trace.summarise_rounds(str(path), sm_mhz=1000.0)
    assert "rounds traced: 6, cycles ended: 1; columns taken 26, moved 3" in out
    assert "several columns: 5 rounds, median 0.70 us: to the steps 0.60, to the end 0.20 where one moves, 0.10" in out
    assert "one column alone: 1 rounds, median 0.80 us" in out
