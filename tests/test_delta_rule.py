"""When requests go through the chunk kernels of the delta rule: the estimate against timings of both kernels."""

import pytest

from freetoken_b200.parts.delta import chunks_pay


@pytest.mark.parametrize("lens,heads,dim,vdim,tokens_us,chunks_us", [
    ([80], 48, 128, 128, 43, 44), ([96], 48, 128, 128, 51, 46), ([512], 48, 128, 128, 227, 120), ([80], 16, 128, 128, 29, 32),
    ([96], 16, 128, 128, 35, 32), ([96], 16, 64, 64, 32, 28), ([128] * 2, 48, 128, 128, 88, 79), ([128] * 8, 16, 128, 128, 88, 107),
    ([256] * 4, 32, 128, 128, 162, 177), ([256] * 4, 48, 128, 64, 162, 175), ([512] * 4, 48, 128, 128, 608, 427),
    ([128] * 32, 48, 128, 128, 880, 949), ([256] * 16, 16, 64, 64, 156, 177), ([512] * 8, 16, 64, 64, 195, 173),
    ([256] * 8, 48, 128, 80, 463, 345), ([2048], 48, 128, 16, 563, 316)])
def test_the_faster_kernel_is_named(lens, heads, dim, vdim, tokens_us, chunks_us):
    assert chunks_pay(lens, False, heads, dim, vdim) == (chunks_us < tokens_us)
