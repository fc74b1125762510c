"""The tcgen05 attention of prompt portions with kept keys, gates and sinks, and over latent rows,
against float64 and the warp-level kernel."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# (rows, lengths), window, keep_first: tiles of 128 rows and blocks of 64 keys with every remainder,
# portions behind cached keys, a request without keys, kept keys in the window's block and ahead of it
CASES = [
    (([1], [1]), 0, 0),
    (([128, 1, 129], [128, 64, 193]), 0, 0),
    (([300, 0, 77], [300, 0, 500]), 0, 0),
    (([260, 64], [260, 640]), 100, 0),
    (([400, 130], [400, 1000]), 128, 70),
    (([257], [700]), 64, 300),
    (([90, 200], [90, 350]), 33, 5),
]


@pytest.mark.parametrize("page", [8, 16, 128])
@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("dim", [64, 128, 256])
def test_wide_attention(dim, case, page):
    from ayaka_b200.kernels import gemm_tc, ops

    (rows, lengths), window, keep = case
    latent = dim == 256
    heads, kv_heads = (3, 1) if latent else (4, 2)
    g = torch.Generator("cuda").manual_seed(dim + sum(rows) + page)
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    n, scale = sum(rows), 1.5 / math.sqrt(dim)
    q, gate, sink = randn(n, heads * dim).bfloat16(), randn(n, heads * dim), randn(heads)
    pages = [-(-length // page) for length in lengths]
    width = max(pages)
    order = torch.randperm(sum(pages), generator=g, device="cuda").int() + 1
    table = torch.zeros(len(rows), width, dtype=torch.int32, device="cuda")
    nan = float("nan")  # whatever lies behind a request's last key or in pages that are gone
    k_pages = torch.full((sum(pages) + 2, kv_heads, page, dim), nan, device="cuda").bfloat16()
    v_pages = k_pages if latent else k_pages.clone()
    keys, values, at = [], [], 0
    for b, length in enumerate(lengths):
        mine = order[at:at + pages[b]]
        table[b, :pages[b]] = mine
        at += pages[b]
        k = randn(length, kv_heads, dim).bfloat16()
        v = k if latent else randn(length, kv_heads, dim).bfloat16()
        keys.append(k)
        values.append(v)
        # keys that no row of this step sees any more
        gone = max(0, length - rows[b] - window + 1) if window else 0
        for p in range(length):
            if keep <= p < gone:
                continue
            k_pages[mine[p // page], :, p % page] = k[p]
            v_pages[mine[p // page], :, p % page] = v[p]
    starts = torch.tensor([0, *rows]).cumsum(0).int().cuda()
    for gated, sunk in ((False, False), (True, True)):
        outs = []
        for kernel in ("wide", "mma"):
            out = torch.full((n + 1, heads * dim), nan, device="cuda").bfloat16()
            ops.attention_prefill(q, k_pages, v_pages, table, starts,
                                  torch.tensor(lengths).int().cuda(), out, num_heads=heads,
                                  scale=scale, host_rows=rows, window=window, keep_first=keep,
                                  gate=gate if gated else None, sink=sink if sunk else None,
                                  kernel=kernel)
            gemm_tc.check_status(q.device)
            assert torch.isnan(out[n:].float()).all()
            outs.append(out[:n].double())
        first = 0
        for b, (count, length) in enumerate(zip(rows, lengths)):
            mine = slice(first, first + count)
            pos = torch.arange(length - count, length, device="cuda")[:, None]
            key = torch.arange(length, device="cuda")
            seen = (key <= pos) & ((key > pos - window) | (key < keep)) if window else key <= pos
            for h in range(heads):
                kv = h * kv_heads // heads
                s = q[mine, h * dim:(h + 1) * dim].double() @ keys[b][:, kv].double().T * scale
                s = s.masked_fill(~seen, -math.inf)
                if sunk:
                    s = torch.cat([s, sink[h].double().expand(count, 1)], 1)
                want = torch.softmax(s, 1)[:, :length] @ values[b][:, kv].double()
                part = slice(h * dim, (h + 1) * dim)
                if gated:
                    want = want * torch.sigmoid(gate[mine, part].double())
                # probabilities are rounded to bfloat16 (2^-9 of each) and the result once more
                for got in outs:
                    assert (got[mine, part] - want).norm() <= 2.0 ** -7 * want.norm()
            first += count
        # both kernels round the same things: no further apart than either is from float64
        assert (outs[0] - outs[1]).norm() <= 2.0 ** -7 * outs[1].norm()


def test_far_references():
    """Scores whose maximum rises block by block far beyond the running reference, and rows of
    scores far below zero."""
    from ayaka_b200.kernels import gemm_tc, ops

    n, dim = 320, 128
    unit = torch.nn.functional.normalize(torch.randn(dim, device="cuda"), dim=0)
    for sign in (1.0, -1.0):
        rise = torch.linspace(0.0, 12.0, n, device="cuda")[:, None]
        k = (sign * rise * unit + 0.05 * torch.randn(n, dim, device="cuda")).bfloat16()
        q = (6.0 * unit + 0.05 * torch.randn(n, dim, device="cuda")).bfloat16()
        v = torch.randn(n, dim, device="cuda").bfloat16()
        k_pages, v_pages = (torch.cat([torch.zeros(1, 1, 16, dim, device="cuda").bfloat16(),
                                       x.view(-1, 1, 16, dim)]) for x in (k, v))
        table = torch.arange(1, n // 16 + 1, dtype=torch.int32, device="cuda").view(1, -1)
        out = torch.zeros(n, dim, dtype=torch.bfloat16, device="cuda")
        ops.attention_prefill(q, k_pages, v_pages, table, torch.tensor([0, n]).int().cuda(),
                              torch.tensor([n]).int().cuda(), out, num_heads=1, scale=1.0,
                              host_rows=[n], kernel="wide")
        gemm_tc.check_status(out.device)
        s = (q.double() @ k.double().T).masked_fill(
            torch.ones(n, n, device="cuda").triu(1).bool(), -math.inf)
        want = torch.softmax(s, 1) @ v.double()
        assert (out.double() - want).norm() <= 2.0 ** -7 * want.norm()


@pytest.mark.parametrize("kernel,dim", [("wide", 64), ("wide", 128), ("wide", 256),
                                        ("tcgen05", 64)])
def test_short_walks_one_after_another(kernel, dim):
    """Walks of one block up to two rings of blocks, in many more CTAs than fit at one time, so that a
    CTA's shared memory is the next one's as soon as it has left: the bits of a launch alone."""
    from ayaka_b200.kernels import gemm_tc, ops

    page, heads = 64, 16
    latent = dim == 256
    kv_heads = 1 if latent else heads
    rows = [2 + 67 * b for b in range(8)] * 6
    g = torch.Generator("cuda").manual_seed(dim)
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda").bfloat16()  # noqa: E731
    counts = [-(-n // page) for n in rows]
    table = torch.zeros(len(rows), max(counts), dtype=torch.int32, device="cuda")
    at = 1
    for b, count in enumerate(counts):
        table[b, :count] = torch.arange(at, at + count)
        at += count
    k_pages = randn(at, kv_heads, page, dim)
    v_pages = k_pages if latent else randn(at, kv_heads, page, dim)
    q = randn(sum(rows), heads * dim)

    def run(first, last):
        own = slice(sum(rows[:first]), sum(rows[:last]))
        out = torch.zeros_like(q[own])
        lengths = torch.tensor(rows[first:last]).int().cuda()
        starts = torch.tensor([0, *rows[first:last]]).cumsum(0).int().cuda()
        ops.attention_prefill(q[own], k_pages, v_pages, table[first:last], starts, lengths, out,
                              num_heads=heads, scale=dim ** -0.5, host_rows=rows[first:last],
                              kernel=kernel)
        gemm_tc.check_status(out.device)
        return out

    whole = run(0, len(rows))
    assert torch.equal(whole, torch.cat([run(b, b + 1) for b in range(len(rows))]))


@pytest.mark.parametrize("dim,page,more", [
    (96, 16, {}), (256, 16, {}), (128, 4, {}), (128, 24, {}), (128, 16, {"scale": 0.0}),
    (64, 16, {"scores": "sigmoid"}), (128, 16, {"gate": "aside"})])
def test_a_kernel_that_is_asked_for_runs_or_says_so(dim, page, more):
    """What the wide kernel does not serve: an error for who asks for it, another kernel (with no
    launch counted for the first) for who does not."""
    from ayaka_b200.errors import BackendError
    from ayaka_b200.kernels import gemm_tc, ops

    n, heads = 192, 2
    pages = -(-n // page)
    q = torch.randn(n, heads * dim, device="cuda").bfloat16()
    k_pages, v_pages = (torch.randn(pages + 1, 1, page, dim, device="cuda").bfloat16()
                        for _ in range(2))
    table = torch.arange(1, pages + 1, dtype=torch.int32, device="cuda").view(1, -1)
    if more.get("gate"):  # rows of raw gates that do not start on 16 bytes
        more = {"gate": torch.randn(n, heads * dim + 1, device="cuda")[:, 1:]}
    args = dict(num_heads=heads, host_rows=[n], **{"scale": dim ** -0.5, **more})
    tensors = (q, k_pages, v_pages, table, torch.tensor([0, n]).int().cuda(),
               torch.tensor([n]).int().cuda())
    out, plain = (torch.full_like(q, 3.0) for _ in range(2))
    before = ops.launch_count()
    with pytest.raises(BackendError):
        ops.attention_prefill(*tensors, out, kernel="wide", **args)
    assert torch.all(out == 3.0) and ops.launch_count() == before
    ops.attention_prefill(*tensors, out, **args)
    assert ops.launch_count() == before + 1
    ops.attention_prefill(*tensors, plain, kernel="mma", **args)
    gemm_tc.check_status(out.device)
    assert torch.equal(out, plain)
