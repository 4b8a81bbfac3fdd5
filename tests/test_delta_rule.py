"""When requests go through the chunk kernels of the delta rule: the estimate against timings of both kernels."""

import pytest
import torch

from freetoken_b200.kernels import ops
from freetoken_b200.parts.delta import chunks_pay


@pytest.mark.parametrize("lens,heads,kv,dim,vdim,tokens_us,chunks_us", [
    ([80], 24, 12, 64, 64, 26.7, 29.9), ([80], 4, 1, 64, 64, 25.9, 28.9), ([80], 16, 4, 64, 64, 26.2, 27.4), ([80] * 8, 32, 16, 64, 32, 39.7, 55.1),
    ([96] * 16, 48, 48, 64, 48, 129, 228), ([96] * 32, 24, 24, 64, 80, 207, 313), ([96] * 32, 32, 32, 128, 32, 237, 256),
    ([192] * 16, 48, 24, 64, 32, 179, 205), ([192] * 8, 32, 32, 128, 16, 72.6, 79.6), ([80] * 32, 16, 8, 64, 80, 123, 183),
    ([96], 48, 8, 128, 128, 50, 36), ([512], 48, 8, 128, 128, 224, 72), ([96], 24, 6, 128, 64, 31.9, 28.5), ([192] * 32, 16, 4, 64, 80, 281, 183),
    ([256] * 8, 48, 48, 128, 64, 310, 182), ([2048] * 8, 16, 2, 128, 16, 533, 240), ([80] * 16, 32, 4, 128, 256, 361, 241),
    ([96] * 32, 32, 32, 64, 128, 419, 295), ([128] * 32, 32, 16, 64, 48, 216, 176), ([2048] * 2, 32, 32, 64, 48, 568, 250)])
def test_the_faster_kernel_is_named(lens, heads, kv, dim, vdim, tokens_us, chunks_us):
    assert chunks_pay(lens, False, heads, kv, dim, vdim) == (chunks_us < tokens_us)


@pytest.mark.parametrize("sizes", [(64, 1, 4, 2, 128, 64), (1, 1, 4, 2, 64, 16), (33, 2, 48, 8, 128, 128), (65536, 800, 65535, 5, 64, 4096),
                                   (64, 1, 4, 2, 96, 64), (64, 1, 4, 2, 128, 40), (64, 1, 4, 3, 128, 64), (64, 0, 4, 2, 128, 64)])
def test_scratch_is_what_the_library_asks_for(sizes):
    """The same number from both, past 2^31 too, and 0 for sizes that are not taken."""
    assert ops.delta_chunk_scratch(torch.bfloat16, *sizes) == ops._lib().ftk_delta_chunk_scratch(ops.BF16, *sizes)
    assert ops.delta_chunk_scratch(torch.float32, *sizes) == ops._lib().ftk_delta_chunk_scratch(ops.F32, *sizes) == 0
