"""The lane-vector and in-place paths of the operator variants against the general
ones they stand beside: the same inputs through aligned pointers and through
pointers one word off (which take the scalar row kernel and the source
enumeration), inputs that are not reduced, and a stream under capture."""
import numpy as np
import pytest

import fdp
import oracle_lib as orc

pytestmark = pytest.mark.gpu


def _vectors(width, lanes, off, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for n in (orc.main_states(width), orc.main_states(width - 1)) * 2:
        t = torch.randint(-2**31, 2**31 - 1, (n * lanes + off,), dtype=torch.int32, device="cuda", generator=g)
        out.append(t[off:])  # any 32-bit values, not only residues
    return out


@pytest.mark.parametrize("lanes", [1, 2, 3, 5, 8, 13, 16])
@pytest.mark.parametrize("width,p", [(3, 2), (6, 5), (9, 2), (11, 6), (13, 12)])
def test_aligned_and_unaligned_pointers_agree(engine, width, p, lanes):
    import torch
    mods = [(4294967291, 2, 97, 4294966997, 2147483648)[i % 5] for i in range(lanes)]
    got = {}
    for off in (0, 1):
        a, b, c, d = _vectors(width, lanes, 0, 7)
        if off and lanes > 1:
            shift = [torch.empty(t.numel() + 1, dtype=torch.int32, device="cuda")[1:] for t in (a, b, c, d)]
            for s, t in zip(shift, (a, b, c, d)):
                s.copy_(t)
            a, b, c, d = shift
        torch.cuda.synchronize()
        ptrs = [t.data_ptr() for t in (a, b, c, d)]
        engine.reverse2_apply(width, p, mods, *ptrs)
        torch.cuda.synchronize()
        r2 = c.cpu().numpy().copy(), d.cpu().numpy().copy()
        tm = engine.transfer_map(width, p, paired=True)
        tm.apply(mods, *ptrs)
        torch.cuda.synchronize()
        got[off] = (*r2, c.cpu().numpy().copy(), d.cpu().numpy().copy())
        tm.close()
    for x, y in zip(got[0], got[1]):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(got[0][0], got[0][2])  # both are the two cells
    np.testing.assert_array_equal(got[0][1], got[0][3])


def test_reverse2_under_capture(engine):
    import torch
    width, p, mods = 12, 5, [4294967291, 97]
    a, b, c, d = _vectors(width, 2, 0, 3)
    e, f = torch.empty_like(c), torch.empty_like(d)
    torch.cuda.synchronize()
    engine.reverse2_apply(width, p, mods, a.data_ptr(), b.data_ptr(), c.data_ptr(), d.data_ptr())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        engine.reverse2_apply(width, p, mods, a.data_ptr(), b.data_ptr(), e.data_ptr(), f.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(c, e) and torch.equal(d, f)


def test_first_calls_of_a_width_beside_another_streams_capture():
    # What these calls set up on first use (tables, the windows' pool) leaves a
    # capture that runs on another stream alone, also where that is refused to
    # the thread ("global").
    import torch
    with fdp.Engine(0) as eng:
        x = torch.zeros(1024, dtype=torch.int32, device="cuda")
        other = torch.cuda.Stream()
        a, b, c, d = _vectors(13, 1, 0, 5)
        r2 = _vectors(15, 1, 0, 6)[:2]
        r2 = [torch.remainder(t.to(torch.int64), 97).to(torch.int32) for t in r2]
        again = [t.clone() for t in r2]
        mods, wmods = [4294967291], [97]
        w = _vectors(12, 1, 0, 7)
        eng.reverse2_apply(12, 5, mods, *[t.data_ptr() for t in w])  # the library's kernels and count table
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, capture_error_mode="global"):
            x += 1
            eng.reverse2_apply(13, 5, mods, a.data_ptr(), b.data_ptr(), c.data_ptr(), d.data_ptr(), other.cuda_stream)
            eng.apply_cells(15, 14, 1, wmods, r2[0].data_ptr(), r2[1].data_ptr(), other.cuda_stream)
            x += 1
        graph.replay()
        torch.cuda.synchronize()
        assert int(x[0]) == 2
        got = c.clone(), d.clone()
        eng.reverse2_apply(13, 5, mods, a.data_ptr(), b.data_ptr(), c.data_ptr(), d.data_ptr())
        eng.apply_cells(15, 14, 1, wmods, again[0].data_ptr(), again[1].data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(got[0], c) and torch.equal(got[1], d)
        assert torch.equal(r2[0], again[0]) and torch.equal(r2[1], again[1])
