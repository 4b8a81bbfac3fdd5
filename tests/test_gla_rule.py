"""When long portions go as matrix products in gated linear attention: the rule against timings of both ways."""

import pytest

from freetoken_b200.parts import Segment
from freetoken_b200.parts.gla import longest_chunk


@pytest.mark.parametrize("requests,tokens,heads,dim,tokens_us,products_us", [
    (1, 65, 16, 64, 66, 46), (16, 65, 16, 64, 86, 75), (32, 65, 16, 64, 106, 120), (32, 80, 16, 64, 125, 122), (32, 129, 16, 64, 170, 161),
    (16, 65, 64, 64, 167, 190), (32, 65, 64, 64, 310, 359), (32, 129, 64, 64, 523, 505), (32, 65, 16, 128, 332, 304), (32, 65, 48, 128, 867, 814),
    (16, 256, 48, 128, 1242, 788)])
def test_the_faster_way_is_taken(requests, tokens, heads, dim, tokens_us, products_us):
    segments = [Segment(i, i * tokens, tokens, tokens) for i in range(requests)]
    decoding = [Segment(requests + i, requests * tokens + i, 1, 100) for i in range(31)]  # (single chunks go their own way)
    for s in (segments, segments + decoding):
        assert longest_chunk(s, 64, heads, dim) == (64 if products_us < tokens_us else 0)
