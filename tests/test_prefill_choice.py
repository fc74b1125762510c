"""Which kernel serves a step's prompt portions, on the CPU."""

from __future__ import annotations

import pytest

from ayaka_b200.kernels.ops import prefill_kernel


@pytest.mark.parametrize("rows,plain_64,gated_64,dim_128,latent", [
    ([1024], "tcgen05", "wide", "wide", "wide"),
    ([300, 20], "tcgen05", "wide", "wide", "wide"),
    ([256] + [65] * 40, "tcgen05", "wide", "wide", "wide"),
    # the wide tiles of 40 short portions are as many as the narrow ones
    ([256] + [20] * 40, "tcgen05", "mma", "wide", "wide"),
    ([255], "mma", "mma", "wide", "wide"),
    ([127, 60], "mma", "mma", "mma", "mma"),
    ([], "mma", "mma", "mma", "mma"),
])
def test_the_kernel_by_the_steps_rows(rows, plain_64, gated_64, dim_128, latent):
    assert prefill_kernel(rows, 64, 0.1, True, False) == plain_64
    assert prefill_kernel(rows, 64, 0.1, False, False) == gated_64
    for plain in (True, False):
        assert prefill_kernel(rows, 128, 0.1, plain, False) == dim_128
        assert prefill_kernel(rows, 256, 0.1, plain, True) == latent


@pytest.mark.parametrize("dim,same", [(16, False), (96, False), (256, False), (128, True),
                                      (64, True), (192, True)])
def test_what_the_wide_kernel_does_not_serve_goes_past_it(dim, same):
    assert prefill_kernel([1024], dim, 0.1, False, same) == "mma"
    assert prefill_kernel([1024], 128, -0.1, False, False) == "mma"
