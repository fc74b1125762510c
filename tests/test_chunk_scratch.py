"""Which steps the recurrences take in chunks of rows, and the scratch for them, on the CPU."""

from __future__ import annotations

import pytest
import torch

from ayaka_b200.kernels import ops
from ayaka_b200.parts.context import Workspace

WIDE = (64, 128, 64)  # heads, inner, columns of a Mamba-2 layer 2,048 wide


SCANS = {  # a layer's scan at a size (S = 1 and 2, 1, 0.5)
    "mamba2": lambda rows: ops.memory_buffers(rows, 32, 128, 64),
    "wide mamba2": lambda rows: ops.memory_buffers(rows, *WIDE),
    "mlstm": lambda rows: ops.memory_buffers(rows, 4, 256, 256, normed=True),
    "gated": lambda rows: ops.gla_buffers(rows, 8, 128, 256),
    "delta": lambda rows: ops.delta_buffers(rows, 32, 64, 64),
}
PORTIONS = ([1300, 700], [200], [300, 300], [2000, 1, 1], [27000])
# a decode step, short portions, and portions beside so many single rows that these decide
ROW_BY_ROW = ([1] * 64, [63], [10] * 12, [1] * 31 + [64], [1] * 60 + [128], [1] * 200 + [300])


@pytest.mark.parametrize("scan", SCANS)
def test_the_step_alone_says_whether_it_is_taken_in_chunks(scan):
    for rows in PORTIONS:
        assert SCANS[scan](rows) is not None, rows
        assert SCANS[scan](rows)[0] * SCANS[scan](rows)[1] <= ops.MEMORY_MAX_FLOATS
    for rows in ROW_BY_ROW:
        assert SCANS[scan](rows) is None, rows
    assert SCANS[scan]([1 << 20]) is None  # more scratch than there may be
    assert SCANS[scan]([]) is None
    assert ops.delta_buffers([1000], 4, 257, 64) is None


@pytest.mark.parametrize("scan", SCANS)
def test_the_scratch_holds_the_step_and_little_more(scan):
    of = ops.memory_chunks if scan in ("mamba2", "wide mamba2", "mlstm") else ops.linear_chunks
    for rows in PORTIONS:
        assert of(rows) <= SCANS[scan](rows)[0] < 2 * of(rows)


def test_a_spare_buffer_grows_gives_its_memory_back_and_may_be_refused(monkeypatch):
    work = Workspace(512, torch.device("cpu"))
    first = work.spare("chunks", 8, torch.float32, 16)
    assert first.shape == (16, 8) and work.spare("chunks", 8, torch.float32, 3) is first
    grown = work.spare("chunks", 8, torch.float32, 32)
    assert grown.shape == (32, 8) and work.nbytes() == 32 * 8 * 4 and not work._retired
    zeros, room = torch.zeros, 64

    def scarce(shape, **more):
        if shape[0] > room:
            asked.append(shape[0])
            raise torch.OutOfMemoryError("no room")
        return zeros(shape, **more)

    asked: list[int] = []
    monkeypatch.setattr(torch, "zeros", scarce)
    assert work.spare("chunks", 8, torch.float32, 128) is None
    assert work.spare("chunks", 8, torch.float32, 256) is None
    assert asked == [128]  # not asked for again
    assert work.spare("chunks", 8, torch.float32, 64).shape == (64, 8)


def test_what_a_grid_does_not_count_is_left_to_the_scans_row_by_row():
    """The entry points of the chunked scans decline (and launch nothing) where the others serve."""
    from ctypes import c_float, c_int, c_longlong, c_void_p

    from ayaka_b200.kernels.lib import library

    p, z, i, f = c_void_p(4096), c_void_p(0), c_int, c_float
    heads, rows = 70000, 64

    def wide(heads):
        return i(heads * 24)

    recurrent, linear = library("recurrent"), library("linear_attention")
    for heads, rows in ((70000, 64), (60000, 40000)):
        assert recurrent.ayk_mamba2_chunks(
            p, wide(heads), p, i(heads), p, p, z, p, c_longlong(heads * 64), p, p, p, wide(heads),
            i(1), i(rows), i(1), i(heads), i(1), i(8), i(8), p, p, z) == -6
        assert recurrent.ayk_mlstm_chunks(
            p, wide(heads), i(0), i(0), i(0), i(0), z, f(15.0), p, c_longlong(heads * 128), p, p, p,
            wide(heads), i(1), i(rows), i(1), i(heads), i(8), i(8), p, p, z) == -6
    heads = 70000
    assert linear.ayk_gla_chunks(
        p, wide(heads), i(0), i(0), p, wide(heads), f(4.0), f(1.0), p, c_longlong(heads * 64), p, p, p,
        wide(heads), i(1), i(1), i(heads), i(8), i(8), p, z) == -6
    assert linear.ayk_delta_chunks(
        p, wide(heads), i(0), i(0), i(0), p, p, wide(heads), f(0.6), p, c_longlong(heads * 64), p, p,
        p, wide(heads), i(1), i(1), i(heads), i(8), i(8), p, z) == -6
