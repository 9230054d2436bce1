"""COLLATZ_RANGE_STATS=1: the diagnostics form of the range kernel gives the same results and prints what the
launch did and where its warps' cycles went."""
import re

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off,size,k,negative", [((1 << 40) + 12345, 1 << 26, 24, False),   # two words
                                                 ((1 << 60) + 777, 1 << 24, 16, True),      # three
                                                 ((1 << 90) + 777, 1 << 24, 20, False),     # four
                                                 (0, 1 << 17, 24, False)])                  # integers below 2^k
def test_stats_line(verifier, monkeypatch, capfd, off, size, k, negative):
    v = verifier(26)
    want = v.verify_range(off, size, k, negative=negative)
    monkeypatch.setenv("COLLATZ_RANGE_STATS", "1")
    capfd.readouterr()
    got = v.verify_range(off, size, k, negative=negative)
    line = capfd.readouterr().err
    want.device_ms = got.device_ms
    assert got == want
    assert line.startswith("collatz range stats: ")
    counts, cycles = [{a: int(b) for a, b in re.findall(r"(\w+)=(\d+)", part)} for part in line.split("warp_cycles:")]
    assert set(counts) == {"items", "runs", "entries", "windows", "passes", "screened", "screen_windows", "exact_seeds",
                           "run_pairs", "offers", "scouts"}
    assert set(cycles) == {"windows", "entries", "runs", "screen", "exact", "all"}
    assert all(counts[x] > 0 for x in ("items", "runs", "entries", "screened", "exact_seeds", "run_pairs", "offers"))
    # every seed takes a window or is screened; a warp's pass is at most four windows of 32 lanes
    assert counts["windows"] + counts["screened"] >= got.seeds_checked
    assert counts["windows"] <= counts["passes"] * 4 * 32
    assert counts["screened"] >= counts["exact_seeds"] and counts["offers"] >= 2
    assert 0 < sum(c for a, c in cycles.items() if a != "all") <= cycles["all"]
