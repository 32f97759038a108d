"""The bench record names what was timed: a scan whose regex candidates came from
the literal filter is no speculative walk."""
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

INFO = {"n_groups": 2, "n_context_groups": 0, "last_guesses": 0, "last_guess_hits": 0, "last_events": 0,
        "last_kernel_ms": [0.3, 0.007, 0, 0, 0, 0, 0, 0.36], "last_kcandidates": 65536, "last_fixup_chunks": 0,
        "last_chunks": 149797, "last_rewalk_bytes": 0}


def test_source_of_the_candidates():
    sys.path.insert(0, str(ROOT))
    import bench
    n = 1 << 30
    assert bench.candidate_source(INFO, n) == "literal filter (no group walked)"
    # (scans in several windows keep the phases' times only)
    assert bench.candidate_source(dict(INFO, last_kernel_ms=[0.3, 0.6, 0, 0, 0, 0, 0, 1.0]), n) == "walk"
    assert bench.candidate_source(dict(INFO, last_kernel_ms=[1.7, 0.03, 0, 0, 0, 0, 0, 2.0]), 4 * n).startswith("literal")
    assert "anchored" in bench.candidate_source(dict(INFO, n_context_groups=2), n)


def test_walk_record_of_a_scan_without_a_walk():
    sys.path.insert(0, str(ROOT))
    import bench
    rec = bench.walk_record(INFO, 1 << 30, 0.375)
    assert rec["candidates_from"].startswith("literal filter")
    assert rec["lookups_per_s"] is None and rec["guess_hit_rate"] is None
    walk = dict(INFO, last_guesses=10, last_guess_hits=9, last_kernel_ms=[0, 0.6, 0, 0, 0, 0, 0, 0.8])
    rec = bench.walk_record(walk, 1 << 30, 0.8)
    assert rec["candidates_from"] == "walk" and rec["guess_hit_rate"] == 0.9 and rec["lookups_per_s"] > 0
