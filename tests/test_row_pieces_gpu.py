"""Norms and joins over rows in pieces of four entries against float64, at the widths where the pieces
end: one piece, a piece more or less than a block holds, the most that two pieces a thread and four
hold, and widths and offsets that take the kernels for any row."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

WIDTHS = (4, 252, 1028, 2048, 4096, 4100, 8192, 8196, 1030)
ROWS = 3


def _ops():
    from ayaka_b200.kernels import ops

    return ops


def _randn(*shape, seed=0):
    g = torch.Generator("cuda").manual_seed(seed + shape[-1])
    return torch.randn(*shape, generator=g, device="cuda")


def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    return y if w is None else y * w


def _close(got, want):
    # fp32 sums of up to 8,196 squares and a few products; or one rounding to bfloat16
    tolerance = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2e-6
    assert (got.double() - want).norm() <= tolerance * want.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", WIDTHS)
def test_rms_norm(width, dtype):
    ops = _ops()
    x, z, w = _randn(ROWS, width), _randn(ROWS, width, seed=1), _randn(width, seed=2)
    pick = torch.tensor([2, 0], dtype=torch.int32, device="cuda")
    for mode in ("none", "silu_before", "sigmoid_after", "silu_after"):
        out = torch.zeros(ROWS, width, dtype=dtype, device="cuda")
        gate = {} if mode == "none" else {"gate": z, "gate_mode": mode}
        ops.rms_norm(x, w, 1e-5, out, weight_offset=1.0, count=ROWS, **gate)
        silu = torch.nn.functional.silu(z.double())
        want = _rms(x.double() * (silu if mode == "silu_before" else 1.0), 1.0 + w.double())
        want = want * {"sigmoid_after": torch.sigmoid(z.double()),
                       "silu_after": silu}.get(mode, 1.0)
        _close(out, want)
    out = torch.zeros(2, width, dtype=dtype, device="cuda")
    ops.rms_norm(x, None, 1e-5, out, rows=pick, count=2)
    _close(out, _rms(x.double())[[2, 0]])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", WIDTHS)
def test_norm_add_and_norm_sum(width, dtype):
    ops = _ops()
    # (the second row set starts one entry in: rows that are not whole pieces)
    for shift in (0, 1):
        x, y = (_randn(ROWS, width + 4, seed=s)[:, shift:shift + width] for s in (0, 1))
        start = _randn(ROWS, width, seed=2)
        a, b, c, f = (_randn(width, seed=s) for s in (3, 4, 5, 6))
        dst, copy, out = start.clone(), *(torch.zeros(ROWS, width, dtype=dtype, device="cuda")
                                          for _ in range(2))
        ops.norm_add(x, a, 1e-5, dst, factor=0.7, weight_offset=1.0, copy=copy, rows=ROWS,
                     next_weight=c, next_eps=1e-5, next_offset=1.0, next_out=out, x_factor=0.5,
                     other=y, other_factor=0.9)
        want = start.double() + 0.7 * _rms(0.5 * x.double() + 0.9 * y.double(), 1.0 + a.double())
        _close(dst, want)
        _close(copy, want)
        _close(out, _rms(want, 1.0 + c.double()))
        for accumulate in (True, False):
            dst, out = start.clone(), torch.zeros(ROWS, width, dtype=dtype, device="cuda")
            ops.norm_sum([x, y], [a, b], 1e-5, dst, factor=0.5, scale=f, accumulate=accumulate,
                         rows=ROWS, next_weight=c, next_eps=1e-5, next_out=out)
            want = 0.5 * f.double() * (_rms(x.double(), a.double()) + _rms(y.double(), b.double()))
            want = want + start.double() if accumulate else want
            _close(dst, want)
            _close(out, _rms(want, c.double()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", WIDTHS)
def test_moe_join(width, dtype):
    ops = _ops()
    top, experts = 3, 5
    pair_out, share = _randn(ROWS * top, width), torch.rand(ROWS * top, device="cuda")
    hidden, scale = _randn(ROWS, width, seed=1).to(dtype), _randn(width, seed=2)
    start, c = _randn(ROWS, width, seed=3), _randn(width, seed=4)
    chosen = torch.tensor([0, 5, 2, 4, 1, 3, 6, 5, 0], dtype=torch.int32, device="cuda")
    rows = pair_out.double().view(ROWS, top, width).clone()
    identity = chosen.view(ROWS, top) >= experts
    rows[identity] = hidden.double()[identity.nonzero()[:, 0]]
    pair_out.view(ROWS, top, width)[identity] = float("nan")  # nobody wrote these
    mixed = (share.double().view(ROWS, top, 1) * rows).sum(1) * scale.double()
    for accumulate in (True, False):
        dst, out = start.clone(), hidden.clone()  # the next norm may lie where `hidden` was
        ops.moe_join(pair_out, share, dst, top=top, scale=scale, accumulate=accumulate, rows=ROWS,
                     chosen=chosen, hidden=out, experts=experts, next_weight=c, next_eps=1e-5,
                     next_out=out)
        want = mixed + start.double() if accumulate else mixed
        _close(dst, want)
        _close(out, _rms(want, c.double()))


@pytest.mark.parametrize("width", [4, 1028, 2048, 4100, 1030])
@pytest.mark.parametrize("rows", [127, 128, 300])
def test_joins_of_few_and_of_many_rows(rows, width):
    """Without a next norm the rows of a large step are taken in pieces, those of a small one entry by
    entry: the same bits."""
    ops = _ops()
    top, experts = 3, 4
    pair_out, share = _randn(rows * top, width), torch.rand(rows * top, device="cuda")
    hidden, scale = _randn(rows, width, seed=1).bfloat16(), _randn(width, seed=2)
    chosen = torch.arange(rows * top, device="cuda").int() % (experts + 1)
    start = _randn(rows, width, seed=3)
    for factor in (scale, None):
        whole, parts = start.clone(), start.clone()
        ops.moe_join(pair_out, share, whole, top=top, scale=factor, rows=rows, chosen=chosen,
                     hidden=hidden, experts=experts)
        for first in range(0, rows, 50):
            few = slice(first, min(rows, first + 50))
            pairs = slice(few.start * top, few.stop * top)
            ops.moe_join(pair_out[pairs], share[pairs], parts[few], top=top, scale=factor,
                         rows=few.stop - few.start, chosen=chosen[pairs], hidden=hidden[few],
                         experts=experts)
        assert torch.equal(whole, parts)
