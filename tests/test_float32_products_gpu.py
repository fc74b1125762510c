"""The CUDA-core product by each of its routes against float64: pieces of 16 bytes, of 4 (rows or sums
that are not whole aligned pieces) and 16-bit operands, K in one stretch and over clusters of 2, 4 and
8, tiles of 32 x 32 and of 64 x 64; and that a row's bits do not depend on its batch."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# rows (the second of each pair fills the device with tiles of 64 x 64), columns, K; stretches of K
SHAPES = [
    ((1, 33, 700), 1500, 383, 1), ((5, 2100), 300, 257, 1), ((3, 4800), 130, 384, 2),
    ((7, 2430), 200, 772, 4), ((31, 1300), 70, 1540, 8), ((64, 1290), 96, 3072, 8),
    ((65, 1285), 72, 1541, 8), ((2, 2460), 129, 770, 4), ((4, 4700), 100, 386, 2),
]


def _operands(m, n, k, dtype, shift=0):
    g = torch.Generator("cuda").manual_seed(m + n + k)
    a = torch.randn(m, k + 4, generator=g, device="cuda").to(dtype)[:, shift:shift + k]
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).to(dtype)
    return a, w, torch.randn(n, generator=g, device="cuda"), torch.randn(m, n, generator=g,
                                                                        device="cuda")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n,k,stretches", SHAPES)
def test_every_route_against_float64(rows, n, k, stretches, dtype):
    from ayaka_b200.kernels import ops

    for m in rows:
        for shift in (0, 1):  # the second: rows that start anywhere
            a, w, bias, base = _operands(m, n, k, dtype, shift)
            want = a.double() @ w.double().T + bias.double()
            out, acc = torch.full((m, n), float("nan"), device="cuda"), base.clone()
            ops.linear(a, w, bias, out, kernel="simt")
            ops.linear(a, w, bias, acc, residual=True, kernel="simt")
            # two sums a stretch of up to 192 to 768 terms each, then a stretch after the other
            for got, right in ((out, want), (acc, want + base.double())):
                assert (got.double() - right).norm() <= 2e-6 * want.norm()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n,k,stretches", SHAPES)
def test_a_rows_bits_do_not_depend_on_its_batch(rows, n, k, stretches, dtype):
    from ayaka_b200.kernels import ops

    m = max(rows)
    a, w, bias, _ = _operands(m, n, k, dtype)
    whole = torch.empty(m, n, device="cuda")
    ops.linear(a, w, bias, whole, kernel="simt")
    for first, last in ((0, 1), (m // 2, m // 2 + 40), (m - 1, m)):
        part = torch.empty(last - first, n, device="cuda")
        ops.linear(a[first:last], w, bias, part, kernel="simt")
        assert torch.equal(part, whole[first:last])
