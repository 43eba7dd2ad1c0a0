"""Cells that go run by run against the same cells item by item (lane counts 2 and 4
never take runs at 32-bit ranks), at widths on both sides of the line."""
import numpy as np
import pytest

import fdp
import oracle_lib as orc

pytestmark = pytest.mark.gpu
MODS = [4294967291, 2, 4294966997, 97, 2147483648, 2147483649, 4294967295, 65537]


def _window(engine, width, mods, main, blk, p_hi, p_lo):
    import torch
    dm = torch.from_numpy(fdp.pack_lanes(main).view(np.int32)).cuda()
    db = torch.from_numpy(fdp.pack_lanes(blk).view(np.int32)).cuda()
    engine.apply_cells(width, p_hi, p_lo, mods, dm.data_ptr(), db.data_ptr())
    torch.cuda.synchronize()
    return (fdp.unpack_lanes(dm.cpu().numpy().view(np.uint32), len(main), len(mods)),
            fdp.unpack_lanes(db.cpu().numpy().view(np.uint32), len(blk), len(mods)))


@pytest.mark.parametrize("width", [14, 17, 18])
@pytest.mark.parametrize("lanes", [1, 3, 5, 6, 8])
def test_runs_equal_items(engine, width, lanes):
    rng = np.random.default_rng(width * 16 + lanes)
    cols = [np.stack([rng.integers(0, m, size=n, dtype=np.uint64) for m in MODS[:lanes]], 1).astype(np.uint32)
            for n in (orc.main_states(width), orc.main_states(width - 1))]
    got = _window(engine, width, MODS[:lanes], *cols, width - 1, 8)
    for l in range(0, lanes, 2):
        pair = [l, (l + 1) % lanes]  # an odd count takes its first lane again
        want = _window(engine, width, [MODS[i] for i in pair], *[np.ascontiguousarray(x[:, pair]) for x in cols],
                       width - 1, 8)
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a[:, pair], b)
