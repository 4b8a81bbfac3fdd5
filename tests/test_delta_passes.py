"""The delta rule's chunks in passes over less scratch than all rows take."""

import random

import pytest
import torch

from freetoken_b200.kernels import ops
from freetoken_b200.parts.delta import CHUNK_MIN_TOKENS, chunk_passes


@pytest.mark.parametrize("most", [1, 2, 7, 32, 200])
def test_passes_take_every_row_once_and_in_order(most):
    rng = random.Random(most)
    for lens in [[64], [65], [8192], [80] * 102, [4096] + [80] * 51, [2048] * 4] + [[rng.randint(80, 3000) for _ in range(rng.randint(1, 40))] for _ in range(20)]:
        done = [0] * len(lens)
        for first, count, row0, row1, rows in chunk_passes(lens, most):
            took = 0
            for i in range(first, first + count):
                n = max(0, min(-(-lens[i] // 64), row1) - row0)
                assert n == 0 or done[i] == row0
                done[i] += n
                took += n
            assert 0 < took == rows <= most
        assert done == [-(-n // 64) for n in lens]
    assert chunk_passes([2048] * 4, 128) == [(0, 4, 0, 32, 128)]
    assert chunk_passes([2048] * 4, 64) == [(0, 4, 0, 16, 64), (0, 4, 16, 32, 64)]  # side by side
    assert chunk_passes([8192], 64) == [(0, 1, 0, 64, 64), (0, 1, 64, 128, 64)]
    assert chunk_passes([80, 8192, 65, 64], 64) == [(0, 4, 0, 59, 64), (0, 4, 59, 123, 64), (0, 4, 123, 128, 5)]
    assert chunk_passes([4096] + [80] * 51, 63) == [(0, 1, 0, 63, 63), (0, 1, 63, 64, 1), (1, 31, 0, 2, 62), (32, 20, 0, 2, 40)]
    assert [p[1] for p in chunk_passes([80] * 102, 64)] == [32, 32, 32, 6]  # whole: a state is read and written once


def test_an_engines_scratch_stays_near_what_it_was():
    """48 heads on 8 of 128: 150 MB for steps of 8,192 tokens and 300 MB for 16,384 before T and A T were kept as the tensor core reads them."""
    from freetoken_b200.config.spec import PartSpec
    from freetoken_b200.parts import MIXERS, BuildEnv, Workspace

    for tokens, most in ((2048, 90e6), (8192, 180e6), (16384, 360e6)):
        env = BuildEnv(dtype=torch.bfloat16, device=torch.device("cpu"), max_seq_len=32768, max_step_tokens=tokens, workspace=Workspace(torch.device("cpu")))
        part = MIXERS.build(PartSpec("gated_delta", dict(hidden=3072, n_heads=48, n_kv_heads=8, head_dim=128, eps=1e-6)), env)
        rows, size = part.chunk_scratch(tokens, tokens // CHUNK_MIN_TOKENS)
        assert 32 <= rows and 0 < size < most
        assert part.chunk_scratch(200, 1) == (4, ops.delta_chunk_scratch(torch.bfloat16, 200, 1, 48, 8, 128, 128))


@pytest.mark.gpu
@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 48), (6, 1, 64, 16), (48, 8, 128, 128)])
@pytest.mark.parametrize("lens", [[(300, 300), (80, 90), (1, 30), (129, 129), (192, 500)], [(1, 9)] * 35 + [(513, 600)] + [(7, 7)] * 3 + [(100, 100)] * 3])
@pytest.mark.parametrize("most", [1, 3, 8])
def test_passes_change_no_bit(H, G, D, Dv, lens, most):
    """States go through their slots between passes, 32 bits as they are."""
    from test_delta_chunks_gpu import EPS, problem, scan

    p = problem(lens, H, G, D, Dv, seed=most)
    long = [n for n, _ in lens if n >= 80]
    want, want_state = scan(p, long_from=80, n_long=len(long))
    row = ops.delta_chunk_scratch(torch.bfloat16, 64, 1, H, G, D, Dv) // 2
    passes = chunk_passes(long, most)
    guarded = torch.full(((most + 1) * row,), 171, dtype=torch.uint8, device="cuda")
    out, state = torch.full_like(want, float("nan")), p["state"].clone()
    before = ops.launch_count()
    ops.delta_scan(p["q"], p["k"], p["v"], p["b"], p["a"], p["a_log"], p["dt_bias"], D ** -0.5, EPS, state, p["slots"], p["info"], len(lens),
                   out, scratch=guarded[:most * row], long_from=80, n_long=len(long), passes=passes)
    assert ops.launch_count() - before == 1 + 2 * len(passes)
    assert torch.equal(out, want) and torch.equal(state, want_state) and bool((guarded[most * row:] == 171).all())
    assert ops.read_status() == 0
