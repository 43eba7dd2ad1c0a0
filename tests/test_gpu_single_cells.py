"""Passes with every cell its own launch (as where no memory is left for the fused
low cells, and at n <= 11 instead of one launch): the same residues as the default
passes, for one and several panels and, above 8 lanes, two span chains."""
import pytest

import fdp
import oracle_lib as orc

pytestmark = pytest.mark.gpu
P = orc.largest_primes_below_2_32(16)


@pytest.fixture
def cells():
    with fdp.Engine(0) as eng:
        eng.single_cells()
        yield eng


@pytest.mark.parametrize("n", list(range(1, 14)))
def test_small_grids_match_oracle_cell_by_cell(cells, n):
    mods = [P[0], 2, 3, 2147483647]
    got = cells.residues(n, mods, lanes=4).residues
    assert got == cells.residues(n, mods, lanes=1).residues
    assert got[:1] == [orc.residue(n, mods[0])]


@pytest.mark.parametrize("n", [12, 13, 16])
@pytest.mark.parametrize("lanes", [2, 5, 7, 9, 14, 16])
def test_lane_counts_agree_cell_by_cell_and_fused(engine, cells, n, lanes):
    want = engine.residues(n, P, lanes=1).residues
    assert cells.residues(n, P, lanes=lanes).residues == want  # from 9 lanes on: two chains
    assert engine.residues(n, P, lanes=lanes).residues == want


def test_launches_tell_the_paths_apart(engine, cells):
    for n in (9, 16):
        one, many = engine.residues(n, P[:2], 2), cells.residues(n, P[:2], 2)
        assert one.residues == many.residues and one.stats.kernel_launches < many.stats.kernel_launches


def test_several_problems_cell_by_cell(engine, cells):
    problems = [(9, P[:3]), (14, P[3:7]), (12, [2, 3, 5]), (16, P[:14])]
    assert cells.residues_multi(problems)[0] == engine.residues_multi(problems)[0]


def test_windows_cell_by_cell(engine, cells):
    import torch
    width, mods = 15, P[:3]
    g = torch.Generator(device="cuda").manual_seed(2)
    main, blk = (torch.randint(0, 2**31 - 1, (3 * n,), dtype=torch.int32, device="cuda", generator=g)
                 for n in (orc.main_states(width), orc.main_states(width - 1)))
    other = main.clone(), blk.clone()
    torch.cuda.synchronize()
    engine.apply_cells(width, 14, 1, mods, main.data_ptr(), blk.data_ptr())
    cells.apply_cells(width, 14, 1, mods, other[0].data_ptr(), other[1].data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(main, other[0]) and torch.equal(blk, other[1])
