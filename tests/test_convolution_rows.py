"""The short convolution by one and by eight rows a thread: which step takes which, and both against
float64."""

from __future__ import annotations

from ctypes import c_int

import pytest
import torch


@pytest.mark.parametrize("rows,requests,channels,each", [
    (1, 1, 2304, 1), (8, 8, 2304, 1), (256, 256, 4352, 1),  # decode steps
    (64, 1, 4352, 1), (80, 17, 100000, 1),                  # few rows, or few a request
    (228, 1, 2304, 8), (2324, 2, 2304, 8), (4096, 256, 2304, 8), (4096, 257, 2304, 1)])
def test_few_rows_have_a_thread_each(rows, requests, channels, each):
    from ayaka_b200.kernels.lib import library

    got = library("recurrent").ayk_causal_conv_rows(c_int(rows), c_int(requests), c_int(channels))
    assert got == each


# portions that start and end anywhere in a stretch of eight rows, single rows, padding rows
@pytest.mark.gpu
@pytest.mark.parametrize("taps", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("rows,channels,each", [([3, 61, 1, 58, 47], 3300, 8), ([300], 1800, 8),
                                                ([1, 1, 1, 1, 1], 300, 1), ([3, 30, 25], 70, 1)])
def test_the_convolution_of_portions(rows, channels, each, taps):
    from ayaka_b200.kernels import ops
    from ayaka_b200.kernels.lib import library

    total, requests = sum(rows), len(rows)
    assert library("recurrent").ayk_causal_conv_rows(c_int(total), c_int(requests),
                                                     c_int(channels)) == each
    g = torch.Generator("cuda").manual_seed(total + taps)
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    x, weight, bias = randn(total, channels), randn(channels, taps), randn(channels)
    state = randn(requests + 1, (taps - 1) * channels + 4)
    kept, out = state.clone(), torch.full((total, channels), 7.0, device="cuda")
    req = torch.cat([torch.full((n,), b) for b, n in enumerate(rows)]).int().cuda()
    pad = total // 2
    req[pad] = -1  # a padding row: nothing is written
    ops.causal_conv_silu(x, weight, bias, state, out, request_of_row=req,
                         row_start=torch.tensor([0, *rows]).cumsum(0).int().cuda(),
                         state_slot=torch.arange(requests, 0, -1).int().cuda(), rows=total,
                         requests=requests)
    first = 0
    for b, n in enumerate(rows):
        slot = requests - b
        before = kept[slot, :(taps - 1) * channels].view(taps - 1, channels)
        u = torch.cat([before, x[first:first + n]]).double()
        want = sum((u[i:i + n] * weight[:, i].double() for i in range(taps)), bias.double())
        want = torch.nn.functional.silu(want)
        for t in range(n):
            if first + t == pad:
                assert torch.all(out[pad] == 7.0)
            else:  # fp32 sums of up to eight terms
                assert (out[first + t].double() - want[t]).norm() <= 1e-6 * want[t].norm()
        moved = state[slot, :(taps - 1) * channels].view(taps - 1, channels)
        assert torch.equal(moved, u[n:].float())
        assert torch.equal(state[slot, (taps - 1) * channels:], kept[slot, (taps - 1) * channels:])
        first += n
    assert torch.equal(state[0], kept[0])
