"""Mamba-2, mLSTM, gated linear attention and the generalised delta rule taken in chunks of rows against
the recurrences in float64: several requests of any length in one step, states that go on from one,
sizes with remainders of every tile, rows that are no numbers."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = ([200, 1, 64, 65], [130], [64, 0, 127])  # whole chunks, single rows, a row behind a chunk
# relative 2-norm; fp32 sums of up to 512 terms and products of up to 200 factors
TOLERANCE = 2e-6


def _step(rows):
    starts = torch.tensor([0, *rows]).cumsum(0).to(torch.int32).cuda()
    slots = torch.arange(len(rows), 0, -1, dtype=torch.int32).cuda()  # slot 0 stays unused
    return dict(row_start=starts, state_slot=slots, requests=len(rows), host_rows=rows)


def _scratch(rows, heads, inner, columns, planes):
    from ayaka_b200.kernels import ops

    nan = float("nan")  # whatever an earlier layer left there
    return (torch.full((ops.memory_chunks(rows), heads * inner * (columns + 1)), nan,
                       device="cuda"), torch.full((sum(rows), planes * heads), nan, device="cuda"))


def _walk(rows, state, decay, take, q, k, v):
    """``S = g S + m k v^T``, ``S^T q`` per request; state [slots, heads, columns, inner]."""
    out, first = torch.zeros_like(v), 0
    for b, count in enumerate(rows):
        S = state[len(rows) - b]
        for t in range(first, first + count):
            S = decay[t, :, None, None] * S + \
                take[t, :, None, None] * v[t, :, :, None] * k[t, :, None, :]
            out[t] = (S @ q[t, :, :, None])[..., 0]
        state[len(rows) - b] = S
        first += count
    return out


def _close(got, want, tolerance=TOLERANCE):
    assert (got.double() - want).norm() <= tolerance * want.norm()


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("heads,groups,inner,columns", [(4, 2, 16, 16), (2, 1, 132, 68),
                                                        (3, 3, 64, 64), (2, 2, 40, 128),
                                                        (150, 50, 20, 12)])
def test_mamba2_in_chunks(heads, groups, inner, columns, rows):
    from ayaka_b200.kernels import ops

    g = torch.Generator("cuda").manual_seed(inner + sum(rows))
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    total, width = sum(rows), heads * columns
    xbc, dt_raw = 0.7 * randn(total, width + 2 * groups * inner), randn(total, heads)
    dt_raw[::7] = 40.0  # a head that forgets everything at once
    dt_bias, a_log, skip = randn(heads), randn(heads), randn(heads)
    state = randn(len(rows) + 1, heads * inner * columns)
    wide = state.double().view(-1, heads, columns, inner)
    x, B, C = xbc.double().split([width, groups * inner, groups * inner], 1)
    B, C = (part.reshape(total, groups, inner).repeat_interleave(heads // groups, 1)
            for part in (B, C))
    x = x.reshape(total, heads, columns)
    dt = torch.nn.functional.softplus(dt_raw.double() + dt_bias.double())
    want = _walk(rows, wide, torch.exp(-torch.exp(a_log.double()) * dt), dt, C, B, x) + \
        skip.double()[:, None] * x
    y = torch.zeros(total, width, device="cuda")
    before = ops.launch_count()
    ops.mamba2_scan(xbc, dt_raw, dt_bias, a_log, skip, state, y, heads=heads, groups=groups,
                    state_size=inner, columns=columns,
                    scratch=_scratch(rows, heads, inner, columns, 2), **_step(rows))
    assert ops.launch_count() - before == 3  # not row by row
    _close(y, want.flatten(1))
    _close(state, wide.flatten(1))


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("heads,inner,columns", [(3, 16, 20), (2, 132, 68), (1, 256, 128),
                                                 (150, 20, 12)])
def test_mlstm_in_chunks(heads, inner, columns, rows):
    from ayaka_b200.kernels import ops

    g = torch.Generator("cuda").manual_seed(inner + sum(rows))
    total, qk, width, cap = sum(rows), heads * inner, heads * columns, 15.0
    proj = torch.randn(total, 2 * qk + 2 * width + 2 * heads, generator=g, device="cuda")
    proj[:, -2 * heads:] *= 6.0
    if proj.shape[1] % 4:  # rows of whole 16-byte pieces, which the chunked path needs
        proj = torch.nn.functional.pad(proj, (0, 4 - proj.shape[1] % 4))
    gate_at = 2 * qk + 2 * width
    bias = torch.randn(2 * heads, generator=g, device="cuda")
    tiles = -(-columns // 16)
    floats = ops.scan_state_floats("mlstm", heads=heads, inner=inner, columns=columns)
    state = torch.zeros(len(rows) + 1, floats, device="cuda")
    size = heads * inner * columns
    wide = torch.randn(len(rows) + 1, heads, columns, inner, generator=g, device="cuda")
    norm = torch.randn(len(rows) + 1, heads, 1, inner, generator=g, device="cuda")
    most = torch.rand(len(rows) + 1, heads, generator=g, device="cuda")
    state[:, :size] = wide.flatten(1)
    state[:, size:size + heads * tiles * inner] = norm.expand(-1, -1, tiles, -1).flatten(1)
    state[:, size + heads * tiles * inner:size + heads * tiles * (inner + 1)] = \
        most[:, :, None].expand(-1, -1, tiles).flatten(1)
    wide, norm, most = wide.double(), norm.double(), most.double()
    q, k = (proj[:, i * qk:(i + 1) * qk].double().reshape(total, heads, inner) for i in (0, 1))
    v = proj[:, 2 * qk:2 * qk + width].double().reshape(total, heads, columns)
    z = proj[:, gate_at:gate_at + 2 * heads].double() + bias.double()
    z = cap * torch.tanh(z / cap)
    gate, forget = z[:, :heads], torch.nn.functional.logsigmoid(z[:, heads:])
    keep, take, floor = (torch.zeros_like(gate) for _ in range(3))
    first = 0
    for b, count in enumerate(rows):
        m = most[len(rows) - b]
        for t in range(first, first + count):
            new = torch.maximum(forget[t] + m, gate[t])
            keep[t], take[t], floor[t] = torch.exp(forget[t] + m - new), \
                torch.exp(gate[t] - new), torch.exp(-new)
            m = new
        most[len(rows) - b] = m
        first += count
    q = q * inner ** -0.5
    below = _walk(rows, norm, keep, take, q, k, torch.ones_like(v[..., :1])).abs()
    want = _walk(rows, wide, keep, take, q, k, v) / (torch.maximum(below, floor[..., None]) + 1e-6)
    args = dict(heads=heads, dim=inner, columns=columns, k_offset=qk, v_offset=2 * qk,
                i_offset=gate_at, f_offset=gate_at + heads, cap=cap, **_step(rows))
    beside, state_beside = torch.zeros(total, width, device="cuda"), state.clone()
    ops.mlstm_scan(proj, bias, state_beside, beside, **args)  # without scratch: row by row
    out = torch.zeros(total, width, device="cuda")
    before = ops.launch_count()
    ops.mlstm_scan(proj, bias, state, out, scratch=_scratch(rows, heads, inner, columns, 3), **args)
    assert ops.launch_count() - before == 3  # not row by row
    # A factor's exponent, a difference of maxima of 8 to 16, is off by half a unit in the last place
    # of each, and up to 200 factors multiply: both ways' error, so that the one may be as far from
    # float64 as the other and half as much again. Every entry counts, times its denominator: where that
    # cancels, its error is divided by little and would be all that is seen.
    def off(got, right, weight=1.0):
        return float(((got.double() - right) * weight).norm() / (right * weight).norm())

    want, below = want.flatten(1), below.expand(-1, -1, columns).flatten(1)
    parts = [(slice(0, size), wide.flatten(1)),
             (slice(size, size + heads * tiles * inner),
              norm.expand(-1, -1, tiles, -1).flatten(1))]
    assert off(out, want, below) <= 1.5 * off(beside, want, below) + TOLERANCE
    for part, right in parts:
        assert off(state[:, part], right) <= 1.5 * off(state_beside[:, part], right) + TOLERANCE
    got = state[:, size + heads * tiles * inner:size + heads * tiles * (inner + 1)]
    torch.testing.assert_close(got.double(), most[:, :, None].expand(-1, -1, tiles).flatten(1),
                               rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("heads,inner,columns", [(3, 16, 20), (2, 130, 33), (1, 128, 256),
                                                 (2, 65, 7)])
def test_gated_linear_attention_in_chunks(heads, inner, columns, rows):
    from ayaka_b200.kernels import ops

    g = torch.Generator("cuda").manual_seed(inner + sum(rows))
    total, qk, width = sum(rows), heads * inner, heads * columns
    proj = torch.randn(total, 2 * qk + width + 3, generator=g, device="cuda")
    z = 3.0 * torch.randn(total, qk, generator=g, device="cuda") + 2.0
    z[::9] = -300.0  # channels that forget everything at once
    state = torch.randn(len(rows) + 1, heads * inner * columns, generator=g, device="cuda")
    wide = state.double().view(-1, heads, columns, inner)
    q, k = (proj[:, i * qk:(i + 1) * qk].double().reshape(total, heads, inner) for i in (0, 1))
    v = proj[:, 2 * qk:2 * qk + width].double().reshape(total, heads, columns)
    decay = torch.exp(torch.nn.functional.logsigmoid(z.double()) / 4.0).view(total, heads, inner)
    want, first = torch.zeros_like(v), 0
    for b, count in enumerate(rows):
        S = wide[len(rows) - b]
        for t in range(first, first + count):
            S = decay[t, :, None, :] * S + v[t, :, :, None] * k[t, :, None, :]
            want[t] = (S @ q[t, :, :, None])[..., 0] * inner ** -0.5
        wide[len(rows) - b] = S
        first += count
    floats = heads * (32 * inner + -(-inner // 4) * 4 + 256)
    scratch = torch.full((ops.linear_chunks(rows), floats), float("nan"), device="cuda")
    out = torch.zeros(total, width, device="cuda")
    before = ops.launch_count()
    ops.gla_scan(proj, z, state, out, heads=heads, dim=inner, columns=columns, k_offset=qk,
                 v_offset=2 * qk, tau=4.0, q_scale=inner ** -0.5, scratch=scratch, **_step(rows))
    assert ops.launch_count() - before == 2  # not row by row
    _close(out, want.flatten(1))
    _close(state, wide.flatten(1))


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("heads,inner,columns", [(3, 16, 20), (2, 130, 33), (2, 64, 64),
                                                 (2, 65, 7), (1, 256, 40)])
def test_generalised_delta_rule_in_chunks(heads, inner, columns, rows):
    from ayaka_b200.kernels import ops

    g = torch.Generator("cuda").manual_seed(inner + sum(rows))
    total, qk, width = sum(rows), heads * inner, heads * columns
    proj = torch.randn(total, 3 * qk + width + 3, generator=g, device="cuda")
    proj[5] = 0.0  # a key of length nothing
    z = 3.0 * torch.randn(total, qk, generator=g, device="cuda")
    bias = torch.randn(qk, generator=g, device="cuda")
    state = torch.randn(len(rows) + 1, heads * inner * columns, generator=g, device="cuda")
    wide = state.double().view(-1, heads, columns, inner)
    r, k, y = (proj[:, i * qk:(i + 1) * qk].double().reshape(total, heads, inner) for i in range(3))
    v = proj[:, 3 * qk:3 * qk + width].double().reshape(total, heads, columns)
    w = torch.exp(-0.6065 * torch.sigmoid(z.double())).view(total, heads, inner)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = torch.sigmoid(y + bias.double().view(heads, inner)) * u
    want, first = torch.zeros_like(v), 0
    for b, count in enumerate(rows):
        S = wide[len(rows) - b]
        for t in range(first, first + count):
            seen = (S @ u[t, :, :, None])[..., 0]
            S = w[t, :, None, :] * S - seen[:, :, None] * au[t, :, None, :] + \
                v[t, :, :, None] * k[t, :, None, :]
            want[t] = (S @ r[t, :, :, None])[..., 0]
        wide[len(rows) - b] = S
        first += count
    floats = heads * (64 * inner + -(-inner // 4) * 4 + 256)
    scratch = torch.full((ops.linear_chunks(rows), floats), float("nan"), device="cuda")
    out = torch.zeros(total, width, device="cuda")
    before = ops.launch_count()
    ops.delta_scan(proj, z, bias, state, out, heads=heads, dim=inner, columns=columns, k_offset=qk,
                   a_offset=2 * qk, v_offset=3 * qk, decay_rate=0.6065, scratch=scratch,
                   **_step(rows))
    assert ops.launch_count() - before == 2  # not row by row
    _close(out, want.flatten(1))
    _close(state, wide.flatten(1))


def _rows_before(run, operands, row, rows):
    """``run(**operands)``: outputs of a step whose request 1 has an infinity, then a NaN, in every
    entry of its row ``row`` of one operand after the other: the request's rows before it and the other
    requests are what they were."""
    first = rows[0] + row
    clean = run(**operands)
    for name, operand in operands.items():
        for value in (float("inf"), -float("inf"), float("nan")):
            bad = operand.clone()
            bad[first] = value
            got = run(**{**operands, name: bad})
            assert torch.equal(got[:first], clean[:first]), (name, value)
            assert torch.equal(got[sum(rows[:2]):], clean[sum(rows[:2]):]), (name, value)


@pytest.mark.parametrize("row", [0, 1, 37, 63, 90])
def test_mamba2_and_mlstm_take_no_later_row_into_an_earlier_one(row):
    from ayaka_b200.kernels import ops

    rows, heads, inner, columns = [70, 130, 66], 2, 36, 68
    g = torch.Generator("cuda").manual_seed(row)
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    total, qk, width = sum(rows), heads * inner, heads * columns
    dt_bias, a_log, skip = randn(heads), randn(heads), randn(heads)

    def mamba2(x, B, C, dt):
        y = torch.zeros(total, width, device="cuda")
        ops.mamba2_scan(torch.cat([x, B, C], 1), dt, dt_bias, a_log, skip,
                        torch.zeros(4, heads * inner * columns, device="cuda"), y, heads=heads,
                        groups=heads, state_size=inner, columns=columns,
                        scratch=_scratch(rows, heads, inner, columns, 2), **_step(rows))
        return y

    _rows_before(mamba2, dict(x=randn(total, width), B=randn(total, qk), C=randn(total, qk),
                              dt=randn(total, heads)), row, rows)
    floats = ops.scan_state_floats("mlstm", heads=heads, inner=inner, columns=columns)

    def mlstm(q, k, v, i, f):
        out = torch.zeros(total, width, device="cuda")
        ops.mlstm_scan(torch.cat([q, k, v, i, f], 1), None,
                       torch.zeros(4, floats, device="cuda"), out, heads=heads, dim=inner,
                       columns=columns, k_offset=qk, v_offset=2 * qk, i_offset=2 * qk + width,
                       f_offset=2 * qk + width + heads, cap=15.0,
                       scratch=_scratch(rows, heads, inner, columns, 3), **_step(rows))
        return out

    _rows_before(mlstm, dict(q=randn(total, qk), k=randn(total, qk), v=randn(total, width),
                             i=randn(total, heads), f=randn(total, heads)), row, rows)


@pytest.mark.parametrize("row", [1, 10, 15, 37, 63, 90])
def test_gated_and_delta_scans_take_no_later_row_into_an_earlier_one(row):
    from ayaka_b200.kernels import ops

    rows, heads, inner, columns = [70, 130, 66], 2, 40, 36
    g = torch.Generator("cuda").manual_seed(row)
    randn = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    total, qk, width = sum(rows), heads * inner, heads * columns
    bias = randn(qk)

    def scratch(floats):
        return torch.full((ops.linear_chunks(rows), heads * (floats * inner + inner + 256)),
                          float("nan"), device="cuda")

    def gated(q, k, v, z):
        out = torch.zeros(total, width, device="cuda")
        ops.gla_scan(torch.cat([q, k, v], 1), z, torch.zeros(4, qk * columns, device="cuda"), out,
                     heads=heads, dim=inner, columns=columns, k_offset=qk, v_offset=2 * qk, tau=4.0,
                     q_scale=0.2, scratch=scratch(32), **_step(rows))
        return out

    def delta(r, k, y, v, z):
        out = torch.zeros(total, width, device="cuda")
        ops.delta_scan(torch.cat([r, k, y, v], 1), z, bias,
                       torch.zeros(4, qk * columns, device="cuda"), out, heads=heads, dim=inner,
                       columns=columns, k_offset=qk, a_offset=2 * qk, v_offset=3 * qk,
                       decay_rate=0.6065, scratch=scratch(64), **_step(rows))
        return out

    operands = dict(k=randn(total, qk), v=randn(total, width), z=randn(total, qk))
    _rows_before(gated, dict(q=randn(total, qk), **operands), row, rows)
    _rows_before(delta, dict(r=randn(total, qk), y=randn(total, qk), **operands), row, rows)
