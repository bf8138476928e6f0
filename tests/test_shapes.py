"""Which tile shape a park's size asks for (exact_ballpark_b200.tiles.shape_for): every shape a one-tile-a-block plan takes,
whole worlds in each tile, few rows spread over many blocks and many rows in full warps."""

import pytest
import torch

from exact_ballpark_b200.tiles import MAX_CAP, SPREAD_WARPS, plan_for, shape_for


@pytest.mark.parametrize("rows", [1, 4, 4 * SPREAD_WARPS, 4 * SPREAD_WARPS + 1, 16 * SPREAD_WARPS + 1, 32 * SPREAD_WARPS,
                                  3 * 148 * 256 - 1, 3 * 148 * 256, 10 ** 7])
@pytest.mark.parametrize("largest", [1, 4, 31, 33, 128, 129, 256, 300, MAX_CAP])
def test_a_shape_fits_its_worlds_and_the_kernels(rows, largest):
    cap, block = shape_for(rows, largest)
    assert largest <= cap <= MAX_CAP and 32 <= block <= 256 and block % 32 == 0
    if largest <= 256:
        assert cap <= block                              # one round a tile
    if rows <= 4 * SPREAD_WARPS and largest <= 4:
        assert (cap, block) == (4, 32)


@pytest.mark.parametrize("sizes", [[4] * 64, [1, 128, 3, 7, 64, 256, 2], [300, 1], [5]])
def test_a_plan_holds_whole_worlds(sizes):
    plan = plan_for(torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes)))
    starts = [sum(sizes[:k]) for k in range(len(sizes) + 1)]
    assert plan.tile_rows[0] == 0 and plan.tile_rows[-1] == starts[-1] and set(plan.tile_rows) <= set(starts)
    assert max(b - a for a, b in zip(plan.tile_rows[:-1], plan.tile_rows[1:])) <= plan.cap
    assert plan_for(torch.tensor([0, 1, 0])) is None
