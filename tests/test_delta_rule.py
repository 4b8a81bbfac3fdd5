"""When requests go through the chunk kernels of the delta rule: the estimate against timings of both kernels."""

import pytest
import torch

from freetoken_b200.kernels import ops
from freetoken_b200.parts.delta import chunks_pay


@pytest.mark.parametrize("lens,heads,dim,vdim,tokens_us,chunks_us", [
    ([80], 48, 128, 128, 43, 44), ([96], 48, 128, 128, 51, 46), ([512], 48, 128, 128, 227, 120), ([80], 16, 128, 128, 29, 32),
    ([96], 16, 128, 128, 35, 32), ([96], 16, 64, 64, 32, 28), ([128] * 2, 48, 128, 128, 88, 79), ([128] * 8, 16, 128, 128, 88, 107),
    ([256] * 4, 32, 128, 128, 162, 177), ([256] * 4, 48, 128, 64, 162, 175), ([512] * 4, 48, 128, 128, 608, 427),
    ([128] * 32, 48, 128, 128, 880, 949), ([256] * 16, 16, 64, 64, 156, 177), ([512] * 8, 16, 64, 64, 195, 173),
    ([256] * 8, 48, 128, 80, 463, 345), ([2048], 48, 128, 16, 563, 316)])
def test_the_faster_kernel_is_named(lens, heads, dim, vdim, tokens_us, chunks_us):
    assert chunks_pay(lens, False, heads, dim, vdim) == (chunks_us < tokens_us)


@pytest.mark.parametrize("sizes", [(64, 1, 4, 2, 128, 64), (1, 1, 4, 2, 64, 16), (33, 2, 48, 8, 128, 128), (65536, 800, 65535, 5, 64, 4096),
                                   (64, 1, 4, 2, 96, 64), (64, 1, 4, 2, 128, 40), (64, 1, 4, 3, 128, 64), (64, 0, 4, 2, 128, 64)])
def test_scratch_is_what_the_library_asks_for(sizes):
    """The same number from both, past 2^31 too, and 0 for sizes that are not taken."""
    assert ops.delta_chunk_scratch(torch.bfloat16, *sizes) == ops._lib().ftk_delta_chunk_scratch(ops.BF16, *sizes)
    assert ops.delta_chunk_scratch(torch.float32, *sizes) == ops._lib().ftk_delta_chunk_scratch(ops.F32, *sizes) == 0
