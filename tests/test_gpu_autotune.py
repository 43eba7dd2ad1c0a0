"""The autotuner scores what a pass runs: passes of one launch (n <= 11), rows with
the low cells fused, a last pass of fewer residues at its own time."""
import pytest

import fdp
import oracle_lib as orc

pytestmark = pytest.mark.gpu
P = orc.largest_primes_below_2_32(16)


def test_a_pass_of_one_launch_is_timed_as_one(engine):
    # Cell by cell the rows of n = 11 take six times as long.
    try:
        best = engine.autotune(11, P[:4], max_lanes=4, repeats=2)["best"]
        engine.residues(11, P[:4], best["lanes"])
        st = engine.residues(11, P[:4], best["lanes"]).stats
        assert 0.4 < best["s_per_residue"] * 4 / st.device_s < 2.0
    finally:
        engine.set_tuning()


def test_the_last_pass_counts_with_its_own_residues(engine):
    try:
        plan = fdp.plan(17, P[:9], 8)
        swept = plan.rows - max(0, plan.init_rows - 1)
        rec = engine.autotune(17, P[:9], max_lanes=8, repeats=1)
        cand = [c for c in rec["candidates"] if c["lanes"] == 8 and "block" in c]
        assert cand
        for c in cand:  # passes of 8 and 1: one lane's row takes a quarter of eight lanes'
            rows = c["s_per_residue"] * 9 * 1e3 / (c["row_ms"] * swept)
            assert c["passes"] == 2 and 1.0 < rows < 1.6
    finally:
        engine.set_tuning()
