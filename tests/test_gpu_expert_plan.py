"""The plan that sorts (token, expert) pairs: experts on both sides of a warp and of a block, runs of no rows, of whole tiles, one more."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


@pytest.mark.parametrize("tile_rows", [128, 256])
@pytest.mark.parametrize("experts", [1, 2, 31, 32, 33, 64, 1023, 1024, 1025])
@pytest.mark.parametrize("tokens,top", [(1, 1), (37, 2), (900, 3)])
def test_plan(experts, tokens, top, tile_rows):
    from llmserver_b200 import ops
    generator = torch.Generator().manual_seed(experts + tokens)
    chosen = torch.randint(0, experts + 2, (tokens, top), generator=generator)      # the last two are identity outputs
    if tokens == 900:
        chosen[:256, 0], chosen[256:513, 0], chosen[:, 1] = 0, experts - 1, min(1, experts - 1)
    plan = ops.moe_plan(chosen.to(torch.int32).to(DEVICE), experts, tile_rows)
    torch.cuda.synchronize()
    counts = torch.bincount(chosen.flatten(), minlength=experts + 2)[:experts].tolist()
    offsets, want = [0], []
    for expert, count in enumerate(counts):
        want += [(expert, offsets[-1] + row, min(tile_rows, count - row)) for row in range(0, count, tile_rows)]
        offsets.append(offsets[-1] + count)
    assert plan.offsets.tolist() == offsets
    tiles = plan.tiles.tolist()
    assert tiles[0] == len(want) and tiles[1:1 + 3 * len(want)] == [number for tile in want for number in tile]
    rows, pairs = plan.row_of_pair.tolist(), plan.pair_of_row.tolist()
    for pair, expert in enumerate(chosen.flatten().tolist()):
        if expert >= experts:
            assert rows[pair] == -1
        else:
            assert offsets[expert] <= rows[pair] < offsets[expert + 1] and pairs[rows[pair]] == pair


def test_plan_of_more_pairs_than_a_block_holds_in_registers():
    test_plan(64, 6000, 3, 256)
