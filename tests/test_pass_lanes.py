"""How many residues a pass holds, by the memory at hand (host logic, CPU only)."""
import pytest

import fdp

GB = 10**9


@pytest.mark.parametrize("n,lanes,have,want", [
    (22, 14, 190 * GB, 8),    # 16.7 GB a lane with escape words: 14 do not fit, 8 do
    (22, 11, 190 * GB, 11),   # 184 GB and the margin fit
    (22, 11, 184 * GB, 8),    # the margin does not
    (22, 14, 131 * GB, 14),   # not even 8: single cells, all lanes in one pass
    (22, 14, 136 * GB, 8),
    (22, 8, 100 * GB, 8),
    (20, 16, 190 * GB, 16),
    (20, 16, 30 * GB, 16),    # below 32 GiB nothing is split
    (21, 16, 60 * GB, 8),
    (12, 16, 1, 16),          # a width without fused rows
    (23, 5, 190 * GB, 5),
])
def test_pass_lanes(n, lanes, have, want):
    assert fdp.lib().fdp_test_pass_lanes(n, lanes, have) == want


def test_pass_lanes_refuses_what_no_pass_has():
    for n, lanes in ((0, 1), (28, 1), (5, 0), (5, 17)):
        assert fdp.lib().fdp_test_pass_lanes(n, lanes, 1 << 40) == 0
