"""Which tiles the experts' grouped products take, on the CPU."""

from __future__ import annotations

import pytest
import torch

from ayaka_b200.kernels import ops


@pytest.mark.parametrize("experts,width,ff,wide_from", [
    # the fewest pairs an expert that take wide tiles: where these were measured to be the faster
    (16, 2048, 2048, 32), (16, 1024, 1024, 32), (64, 1024, 1024, 32), (256, 1024, 256, 32),
    (8, 2048, 2048, 32), (8, 1024, 1024, 64), (4, 1024, 3072, 40), (4, 1024, 1024, 256),
    (8, 512, 512, 512), (2, 512, 512, 2048),
])
def test_wide_tiles_where_they_are_faster(experts, width, ff, wide_from):
    def tile(pairs, dtype=torch.bfloat16):
        return ops.moe_tile_rows(pairs * experts // 2, experts, 2, dtype, width, ff)

    counts = [n for n in (8, 16, 31, 32, 40, 48, 63, 64, 128, 256, 512, 1024, 2048, 4096)]
    for pairs in counts:
        assert tile(pairs) == (128 if pairs >= wide_from else 32), pairs
        assert tile(pairs, torch.float32) == 32
    # without sizes: large experts
    assert ops.moe_tile_rows(16 * experts, experts, 2, torch.bfloat16) == 128
    assert ops.moe_tile_rows(16 * experts - 1, experts, 2, torch.bfloat16) == 32


@pytest.mark.parametrize("experts", [2, 16, 64])
def test_operands_that_tma_does_not_take(experts):
    for pairs, tile in ((32, 32), (63, 32), (64, 128), (1000, 128)):
        assert ops.moe_tile_rows(pairs * experts, experts, 1, torch.bfloat16, 2044, 1020,
                                 tma=False) == tile


@pytest.mark.parametrize("experts", [2, 16, 64])
def test_the_scratch_serves_both_tiles(experts):
    for rows in (1, 33, 700):
        places, tiles = ops.moe_scratch(rows, experts, 2)
        for tile_rows, each in ((32, 1), (128, 2)):
            most = ops.moe_max_tiles(rows, experts, 2, tile_rows)
            assert places >= most * tile_rows and tiles >= most * each
