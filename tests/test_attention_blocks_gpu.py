"""The float32 attention of 32 rows a block against the rows one by one."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [8, 40, 64, 128])
@pytest.mark.parametrize("rows,lengths,window", [
    ([333, 180], [333, 180], 0),                     # a block of two requests
    ([200], [500], 77),
    ([1, 70, 3, 40, 1, 90], [9, 70, 64, 400, 1, 91], 33),
    ([1] * 150 + [64], [5 + i for i in range(150)] + [200], 0),  # single rows: not in blocks
    ([1] * 40 + [2] * 9 + [301], [5 + i for i in range(49)] + [400], 20),  # blocks of single rows
])
def test_float32_attention_in_blocks(rows, lengths, window, dim):
    """Bit for bit what the same rows give a few at a time."""
    from ayaka_b200.kernels import ops

    heads, kv_heads, page = 4, 2, 16
    g = torch.Generator("cuda").manual_seed(dim + len(rows))
    pages = [-(-length // page) for length in lengths]
    shape = (sum(pages) + 1, kv_heads, page, dim)
    k, v = (torch.randn(shape, generator=g, device="cuda") for _ in range(2))
    table = torch.zeros(len(rows), max(pages), dtype=torch.int32, device="cuda")
    at = 1
    for b, count in enumerate(pages):
        table[b, :count] = torch.arange(at, at + count)
        at += count
    req = torch.cat([torch.full((n,), b) for b, n in enumerate(rows)]).int().cuda()
    pos = torch.cat([torch.arange(length - n, length)
                     for n, length in zip(rows, lengths)]).int().cuda()
    req[sum(rows) // 2] = -1  # a padding row
    total = sum(rows)
    assert total > 192
    q = torch.randn(total, heads * dim, generator=g, device="cuda")
    whole, parts = torch.full_like(q, 3.0), torch.full_like(q, 5.0)
    ops.attention(q, k, v, table, req, pos, whole, num_heads=heads, scale=dim ** -0.5, window=window)
    for lo in range(0, total, 50):
        part = slice(lo, min(total, lo + 50))
        ops.attention(q[part], k, v, table, req[part], pos[part], parts[part], num_heads=heads,
                      scale=dim ** -0.5, window=window)
    assert torch.equal(whole, parts)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("order", ["descending", "every second", "twice", "any", "stretches"])
@pytest.mark.parametrize("window", [0, 50])
def test_rows_at_any_positions(order, window, dtype):
    """A request's rows need not be neighbours in the order of their positions: every row against
    float64, and bit for bit what it gives alone."""
    from ayaka_b200.kernels import ops

    heads, kv_heads, page, dim, length, n = 2, 1, 16, 40, 256, 250
    g = torch.Generator("cuda").manual_seed(5)
    k, v = (torch.randn(length // page + 1, kv_heads, page, dim, generator=g, device="cuda").to(dtype)
            for _ in range(2))
    table = torch.arange(1, length // page + 1, dtype=torch.int32, device="cuda").view(1, -1)
    at = torch.arange(n, device="cuda")
    pos = {"descending": n - 1 - at, "every second": 2 * at % length, "twice": at // 2,
           "any": torch.randint(0, length, (n,), generator=g, device="cuda"),
           "stretches": at % 11 + 16 * (at // 11 % 15)}[order].int()
    req = torch.zeros(n, dtype=torch.int32, device="cuda")
    q = torch.randn(n, heads * dim, generator=g, device="cuda").to(dtype)
    whole, alone = torch.full_like(q, 3.0), torch.full_like(q, 5.0)
    ops.attention(q, k, v, table, req, pos, whole, num_heads=heads, scale=dim ** -0.5, window=window)
    for i in range(n):
        one = slice(i, i + 1)
        ops.attention(q[one], k, v, table, req[one], pos[one], alone[one], num_heads=heads,
                      scale=dim ** -0.5, window=window)
    assert torch.equal(whole, alone)
    keys, values = (x[1:].reshape(length, dim).double() for x in (k, v))
    key, last = torch.arange(length, device="cuda"), pos[:, None]
    seen = (key <= last) & ((key > last - window) | (window == 0))
    s = q.double().view(n, heads, dim) @ keys.T * dim ** -0.5
    want = torch.softmax(s.masked_fill(~seen[:, None], -torch.inf), -1) @ values
    # fp32 sums of up to 256 terms, or one rounding to bfloat16
    tolerance = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    assert (whole.double().view_as(want) - want).norm() <= tolerance * want.norm()
