"""Which steps the recurrences take in chunks of rows, and the scratch for them, on the CPU."""

from __future__ import annotations

import pytest
import torch

from ayaka_b200.kernels import ops
from ayaka_b200.parts.context import Workspace

WIDE = (64, 128, 64)  # heads, inner, columns of a Mamba-2 layer 2,048 wide


def test_the_step_alone_says_whether_it_is_taken_in_chunks():
    for rows in ([1300, 700], [64], [100, 1, 1], [28000]):
        for sizes in (ops.memory_buffers(rows, *WIDE), ops.gla_buffers(rows, 16, 128),
                      ops.delta_buffers(rows, 32, 64)):
            assert sizes is not None
            assert sizes[0] * sizes[1] <= ops.MEMORY_MAX_FLOATS
    for rows in ([1] * 64, [63], [64] + [1] * 40, [128 * 64 * 64]):
        assert ops.memory_buffers(rows, *WIDE) is None
    assert ops.delta_buffers([1000], 4, 257) is None


@pytest.mark.parametrize("rows", [[64], [65], [200, 70], [4096], [1300] * 3, [27000]])
def test_the_scratch_holds_the_step_and_little_more(rows):
    for sizes, chunks in ((ops.memory_buffers(rows, *WIDE), ops.memory_chunks(rows)),
                          (ops.gla_buffers(rows, 16, 128), ops.linear_chunks(rows)),
                          (ops.delta_buffers(rows, 32, 64), ops.linear_chunks(rows))):
        assert chunks <= sizes[0] < 2 * chunks


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
