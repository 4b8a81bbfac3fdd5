"""Which attention kernels take which heads, and where a decode step of windowed heads of 64 goes: the rule against timings of both
kernels."""

import pytest
import torch

from freetoken_b200.config.spec import PartSpec
from freetoken_b200.kernels import ops
from freetoken_b200.parts import MIXERS, BuildEnv, Workspace


@pytest.mark.parametrize("heads,kv,n,window,span,mma_us,tc_us", [
    (16, 16, 1, 1024, 2048, 30.7, 26.6), (16, 16, 8, 1024, 2048, 45.1, 41.0), (16, 16, 16, 128, 2048, 28.7, 38.9),
    (16, 16, 64, 512, 2048, 84.0, 114.7), (16, 16, 128, 1024, 2048, 208.9, 260.1), (16, 16, 24, 4096, 8192, 177.1, 159.7),
    (16, 4, 24, 1024, 2048, 41.0, 43.0), (16, 4, 64, 1024, 2048, 61.4, 59.4), (16, 4, 128, 1024, 1024, 57.3, 86.0),
    (32, 8, 8, 512, 2048, 36.8, 34.8), (32, 8, 64, 1024, 2048, 92.2, 112.7), (32, 8, 48, 1024, 2048, 77.8, 73.7),
    (48, 8, 64, 1024, 2048, 96.2, 114.7), (48, 8, 48, 1024, 1024, 59.4, 54.3), (48, 8, 32, 4096, 8192, 170.0, 135.2),
    (16, 2, 48, 1024, 2048, 41.0, 43.0), (16, 2, 8, 128, 2048, 28.7, 28.7)])
def test_windowed_heads_of_64(heads, kv, n, window, span, mma_us, tc_us):
    env = BuildEnv(dtype=torch.bfloat16, device=torch.device("cpu"), max_seq_len=16384, max_step_tokens=256,
                   workspace=Workspace(torch.device("cpu")))
    part = MIXERS.build(PartSpec("gqa_attention", dict(hidden=64, n_heads=heads, n_kv_heads=kv, head_dim=64, eps=1e-6,
                                                       position=PartSpec("none"), window=window)), env)
    assert part.kernel_form(True, n, 16, span) == ((128, False) if tc_us < mma_us else (16, False))


@pytest.mark.parametrize("head_dim", [16, 32, 64, 96, 128, 192, 256])
@pytest.mark.parametrize("page,group", [(16, 1), (16, 128), (16, 129), (8, 4), (64, 6), (24, 4)])
def test_heads_of_the_tensor_core_kernels(head_dim, page, group):
    fits = page % 16 == 0 and group <= 128
    assert ops.attention_tc_fits(head_dim, page, group) == (fits and head_dim == 128)
    assert ops.attention_tc_heads_fit(head_dim, page, group) == (fits and head_dim in (64, 256))
