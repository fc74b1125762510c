"""The experts' grouped products in tiles of 128 pairs (tcgen05, and mma.sync for rows that TMA does
not take) against float64."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# rows, experts, top, width, ff, gated: remainders of the 64 k, 128 / 256 column and 128 pair tiles
CASES = [
    (97, 3, 2, 72, 40, True),      # less than a tile in every direction
    (200, 4, 2, 64, 136, True),    # one column box and eight columns of the next
    (301, 4, 1, 328, 264, False),  # K and N tails of an expert without a gate
    (513, 2, 2, 256, 128, True),   # whole tiles and a single pair behind them
    (700, 5, 2, 1032, 520, True),  # more tiles than a ring, columns of three tiles
    (150, 4, 2, 36, 20, True),     # rows TMA does not take: less than a tile
    (301, 3, 2, 140, 196, True),   # and tiles in every direction with remainders
    (280, 3, 1, 132, 76, False),   # and an expert without a gate
]


@pytest.mark.parametrize("rows,experts,top,width,ff,gated", CASES)
def test_grouped_products(rows, experts, top, width, ff, gated):
    from ayaka_b200.kernels import ops

    g = torch.Generator().manual_seed(rows)
    dev = dict(device="cuda", dtype=torch.bfloat16)
    parts = 2 if gated else 1
    hidden = torch.randn(rows, width, generator=g).to(**dev)
    w_in = (torch.randn(experts * parts * ff, width, generator=g) * width ** -0.5).to(**dev)
    w_out = (torch.randn(experts * width, ff, generator=g) * ff ** -0.5).to(**dev)
    # the last expert gets one pair, identity experts (an index beyond the last) a few
    chosen = torch.stack([torch.randperm(experts - 1, generator=g)[:top] if experts - 1 >= top
                          else torch.arange(top) * 3 for _ in range(rows)])
    chosen[rows // 2, 0] = experts - 1
    chosen[3, top - 1] = experts
    chosen = chosen.to(torch.int32).view(-1).cuda()
    assert ops.moe_tile_rows(rows, experts, top, torch.bfloat16) == 128  # were they large ones
    places, tiles = ops.moe_scratch(rows, experts, top)
    pair_out = torch.full((rows * top, width), float("nan"), device="cuda")
    before = ops.launch_count()
    ops.moe_experts(hidden, w_in, w_out, chosen, pair_out, experts=experts, top=top,
                    limit=7.0, alpha=1.702, shift=1.0, rows=rows, single=not gated, tile_rows=128,
                    sorted_pairs=torch.empty(places, dtype=torch.int32, device="cuda"),
                    tile_expert=torch.empty(tiles, dtype=torch.int32, device="cuda"),
                    inner=torch.full((places, ff), float("nan"), **dev))
    # (the tensor-core products run over a copy of the rows: a launch more)
    assert ops.launch_count() - before == (4 if width % 8 == 0 and ff % 8 == 0 else 3)
    w_in, w_out = w_in.double().view(experts, parts * ff, width), w_out.double()
    for e in range(experts):
        pairs = (chosen == e).nonzero()[:, 0]
        z = hidden[pairs // top].double() @ w_in[e].T
        if gated:
            gate, up = z[:, :ff].clamp(max=7.0), z[:, ff:].clamp(-7.0, 7.0)
            unit = gate * torch.sigmoid(1.702 * gate) * (up + 1.0)
        else:
            unit = torch.relu(z) ** 2
        want = unit.bfloat16().double() @ w_out[e * width:(e + 1) * width].T
        # the unit is rounded to bfloat16 on both sides (2^-9 of an entry); a sum that falls
        # on the other side of a rounding moves a few entries by one more
        assert (pair_out[pairs].double() - want).norm() <= 2.0 ** -8 * want.norm()
