"""Which weights a single token's attention asks for ahead: the rule against timings with and without."""

import pytest
import torch

from freetoken_b200.config.spec import PartSpec
from freetoken_b200.parts import MIXERS, BuildEnv, Workspace


@pytest.mark.parametrize("heads,kv,hidden,span,tokens,with_us,without_us", [
    (48, 8, 3072, 128, 1, 33.2, 34.9), (48, 8, 3072, 512, 1, 35.7, 36.2), (48, 8, 3072, 4096, 1, 39.4, 37.3), (48, 8, 3072, 8192, 1, 43.3, 41.3),
    (32, 8, 4096, 128, 1, 33.4, 34.9), (32, 8, 4096, 512, 1, 35.4, 36.4), (32, 8, 4096, 4096, 1, 39.2, 36.9), (40, 8, 5120, 1024, 1, 45.0, 43.4),
    (40, 8, 5120, 4096, 1, 49.7, 46.5), (64, 8, 8192, 128, 1, 72.3, 64.3), (64, 8, 8192, 2048, 1, 75.2, 66.5), (48, 8, 3072, 2048, 2, 37.2, 35.5)])
def test_the_faster_way_is_taken(heads, kv, hidden, span, tokens, with_us, without_us):
    env = BuildEnv(dtype=torch.bfloat16, device=torch.device("cpu"), max_seq_len=16384, max_step_tokens=64, workspace=Workspace(torch.device("cpu")))
    part = MIXERS.build(PartSpec("gqa_attention", dict(hidden=hidden, n_heads=heads, n_kv_heads=kv, head_dim=128)), env)
    part._step_span, part._step_plan = span, (None,) * 6 + (True,)
    weight = torch.empty(hidden, heads * 128, dtype=torch.bfloat16, device="meta")
    assert bool(part._weight_ahead(tokens, weight)) == (with_us < without_us)
    part._step_plan = (None,) * 6 + (False,)  # (tiles of many rows)
    assert not part._weight_ahead(tokens, weight)
