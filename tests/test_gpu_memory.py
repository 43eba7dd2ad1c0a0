"""Device memory between calls: what a call took beside the state (escape words of
the fused row tail, the problems of a multi-problem call, window words) stands in
nobody's way afterwards, neither this library's calls nor another allocator of
the process."""
import pytest

import fdp
import oracle_lib as orc

pytestmark = pytest.mark.gpu
P = orc.largest_primes_below_2_32(16)
GIB = 1 << 30


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _fill(leave):
    """Device memory that leaves `leave` bytes of the free memory."""
    import torch
    return torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")


def _after_large_pass(eng, n=19, lanes=16):
    # n = 19, 16 lanes: 8.0 GB of state and 3.6 GB of escape words beside it.
    total = _free()
    state = 4 * lanes * (orc.main_states(n + 1) + orc.main_states(n))
    res = eng.residues(n, P[:lanes], lanes).residues
    return total - state, res


def test_another_allocator_gets_what_a_pass_took_beside_its_state():
    import torch
    with fdp.Engine(0) as eng:
        eng.residues(9, P[:1], 1)  # the library's own tables and buffers
        room, _ = _after_large_pass(eng, 20, 8)  # 11.2 GB and 5.1 GB
        x = torch.empty(room - GIB, dtype=torch.uint8, device="cuda")
        del x
        torch.cuda.empty_cache()


def test_server_start_gets_what_a_pass_took_beside_its_state():
    with fdp.Engine(0) as eng:
        eng.residues(9, P[:1], 1)
        room, _ = _after_large_pass(eng)
        eng.server_start(room - GIB, max_active=1, max_lanes=4)
        rid = eng.submit(12, P[:2])
        assert eng.wait(rid)["residues"] == eng.residues(12, P[:2], 1).residues
        eng.server_stop()


def test_multi_and_map_builds_get_what_a_pass_took_beside_its_state():
    import torch
    with fdp.Engine(0) as eng:
        eng.residues(9, P[:1], 1)
        eng.transfer_map(8, 4, paired=False).close()
        _, res = _after_large_pass(eng)
        fill = _fill(GIB)
        # 2.0 GB of state for the multi call; more than 0.5 GB for the map.
        assert eng.residues_multi([(19, P[:4])])[0][0] == res[:4]
        m = eng.transfer_map(19, 9, paired=True)
        assert m.info()["device_bytes"] > 0.5e9
        m.close()
        assert eng.residues(19, P, 16).residues == res  # without room for escape words
        del fill
        torch.cuda.empty_cache()


def test_a_smaller_problem_after_a_larger_one_when_memory_is_short():
    import torch
    with fdp.Engine(0) as eng:
        res = eng.residues(20, P[:8], 8).residues  # leaves 11.2 GB of state buffers
        want = eng.residues(18, P[:1], 1).residues
        fill = _fill(GIB // 2)
        # Escape words of n = 18 (0.65 GB at 8 lanes) fit beside exact buffers alone.
        small = eng.residues(18, P[:8], 8).residues
        del fill
        torch.cuda.empty_cache()
        assert small[:1] == want and small == eng.residues(18, P[:8], 2).residues
        assert eng.residues(20, P[:8], 8).residues == res


def test_another_allocator_gets_what_a_window_left_in_the_pool():
    import torch
    width, mods = 22, P[:1]
    with fdp.Engine(0) as eng:
        a = torch.zeros(orc.main_states(width), dtype=torch.int32, device="cuda")
        b = torch.zeros(orc.main_states(width - 1), dtype=torch.int32, device="cuda")
        eng.apply_cells(12, 11, 1, mods, a.data_ptr(), b.data_ptr())  # the library's own tables
        before = _free()
        eng.apply_cells(width, width - 1, 1, mods, a.data_ptr(), b.data_ptr())
        torch.cuda.synchronize()
        assert _free() < before - GIB  # 1.8 GB of escape words wait for the next window
        x = torch.empty(before - GIB // 2, dtype=torch.uint8, device="cuda")
        del x, a, b
        torch.cuda.empty_cache()


def test_a_second_window_in_flight_leaves_half_of_what_is_free():
    # Windows on two streams, the first held up by a delay: its words (910 MB at
    # width 20, 4 lanes) are not idle although the call that frees them has returned,
    # so the second window's may not be mapped beside them where less than twice as
    # much is free; it runs cell by cell with the same result.
    import torch
    width, mods = 20, P[:4]
    with fdp.Engine(0) as eng:
        g = torch.Generator(device="cuda").manual_seed(1)
        main = torch.randint(0, 2**31 - 1, (4 * orc.main_states(width),), dtype=torch.int32, device="cuda", generator=g)
        blk = torch.randint(0, 2**31 - 1, (4 * orc.main_states(width - 1),), dtype=torch.int32, device="cuda", generator=g)
        pairs = [(main.clone(), blk.clone()), (main, blk)]
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        small = [torch.zeros(n, dtype=torch.int32, device="cuda") for n in (4 * orc.main_states(14), 4 * orc.main_states(13))]
        for s in streams:  # the library's tables and kernels
            eng.apply_cells(14, 13, 1, mods, small[0].data_ptr(), small[1].data_ptr(), s.cuda_stream)
        eng.apply_cells(width, 3, 2, mods, pairs[0][0].data_ptr(), pairs[0][1].data_ptr())
        torch.cuda.synchronize()
        pairs[0][0].copy_(main)
        pairs[0][1].copy_(blk)
        words = int(0.62 * 4 * 4 * orc.main_states(width))
        fill = _fill(5 * words // 2)
        before = torch.cuda.mem_get_info()[0]
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(1_000_000_000)  # half a second
        for s, (a, b) in zip(streams, pairs):
            eng.apply_cells(width, width - 1, 1, mods, a.data_ptr(), b.data_ptr(), s.cuda_stream)
        taken = before - torch.cuda.mem_get_info()[0]
        torch.cuda.synchronize()
        del fill
        torch.cuda.empty_cache()
        assert words // 2 < taken < 3 * words // 2
        assert torch.equal(pairs[0][0], pairs[1][0]) and torch.equal(pairs[0][1], pairs[1][1])


def test_a_row_as_two_windows_takes_no_memory():
    import torch
    width, mods = 20, P[:2]
    with fdp.Engine(0) as eng:
        g = torch.Generator(device="cuda").manual_seed(3)
        main, blk = (torch.randint(0, 2**31 - 1, (2 * n,), dtype=torch.int32, device="cuda", generator=g)
                     for n in (orc.main_states(width), orc.main_states(width - 1)))
        one = main.clone(), blk.clone()
        eng.apply_cells(width, 2, 2, mods, one[0].data_ptr(), one[1].data_ptr())  # the width's tables
        torch.cuda.synchronize()
        one[0].copy_(main)
        one[1].copy_(blk)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        eng.apply_cells(width, width - 1, 2, mods, main.data_ptr(), blk.data_ptr())
        eng.apply_cells(width, 1, 1, mods, main.data_ptr(), blk.data_ptr())
        assert before - torch.cuda.mem_get_info()[0] < 64 << 20  # loaded kernels
        torch.cuda.synchronize()
        eng.apply_cells(width, width - 1, 1, mods, one[0].data_ptr(), one[1].data_ptr())
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] > 400 << 20  # 440 MB of escape words
        assert torch.equal(main, one[0]) and torch.equal(blk, one[1])
