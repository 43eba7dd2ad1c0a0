"""The fused row tail (cells 8..1 of a row in one pass, widths from 14) on the
GPU against the oracle's cells, through the operator window: whole rows and the
window that starts at the tail's first cell, every panel width (lanes 1, 2, 4,
8 and mixed panels), moduli below and above 2^31, and windows on a stream under
capture, which run cell by cell."""
import numpy as np
import pytest

import fdp
import oracle_lib as orc

pytestmark = pytest.mark.gpu
MODS = [4294967291, 2, 4294966997, 97, 2147483648, 2147483649, 4294967295]


def _state(width, mods, seed):
    rng = np.random.default_rng(seed)
    M, D = orc.main_states(width), orc.main_states(width - 1)
    main = np.stack([rng.integers(0, m, size=M, dtype=np.uint64) for m in mods], 1).astype(np.uint32)
    blk = np.stack([rng.integers(0, m, size=D, dtype=np.uint64) for m in mods], 1).astype(np.uint32)
    return M, D, main, blk


def _want(width, p_hi, mods, main, blk):
    om, ob = main.copy(), blk.copy()
    for l, m in enumerate(mods):
        a, b = main[:, l].copy(), blk[:, l].copy()
        for p in range(p_hi, 0, -1):
            a, b = orc.forward_cell(width, p, m, a, b)
        om[:, l], ob[:, l] = a, b
    return om, ob


def _dev(a):
    import torch
    return torch.from_numpy(fdp.pack_lanes(a).view(np.int32)).cuda()


def _host(t, n, lanes):
    return fdp.unpack_lanes(t.cpu().numpy().view(np.uint32), n, lanes)


@pytest.mark.parametrize("width,lanes,p_hi", [(14, 1, 13), (14, 7, 8), (14, 16, 13), (15, 2, 9), (15, 14, 14),
                                              (15, 4, 14), (15, 8, 8), (16, 1, 15)])
@pytest.mark.parametrize("wide", [True, False])
def test_window_down_to_cell_1(engine, width, lanes, p_hi, wide):
    import torch
    mods = [4294967291 if wide and i % 2 else 4294966997 if wide else MODS[i % len(MODS)] for i in range(lanes)]
    M, D, main, blk = _state(width, mods, 31 * width + lanes)
    dm, db = _dev(main), _dev(blk)
    engine.apply_cells(width, p_hi, 1, mods, dm.data_ptr(), db.data_ptr())
    torch.cuda.synchronize()
    want = _want(width, p_hi, mods, main, blk)
    np.testing.assert_array_equal(_host(dm, M, lanes), want[0])
    np.testing.assert_array_equal(_host(db, D, lanes), want[1])


def test_windows_on_two_streams_and_under_capture(engine):
    import torch
    width, mods = 15, [4294967291, 4294966997, 97]
    M, D, main, blk = _state(width, mods, 5)
    want = _want(width, 14, mods, main, blk)
    streams = [torch.cuda.Stream() for _ in range(3)]
    states = [(_dev(main), _dev(blk)) for _ in streams]
    torch.cuda.synchronize()
    for s, (a, b) in zip(streams[:2], states):  # in flight together
        engine.apply_cells(width, 14, 1, mods, a.data_ptr(), b.data_ptr(), s.cuda_stream)
    graph = torch.cuda.CUDAGraph()
    a, b = states[2]
    with torch.cuda.graph(graph, stream=streams[2], capture_error_mode="relaxed"):
        engine.apply_cells(width, 14, 1, mods, a.data_ptr(), b.data_ptr(), torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    for a, b in states:
        np.testing.assert_array_equal(_host(a, M, 3), want[0])
        np.testing.assert_array_equal(_host(b, D, 3), want[1])
