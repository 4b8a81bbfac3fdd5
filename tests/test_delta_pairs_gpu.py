"""The gated delta rule in chunks at the borders of their 64 tokens and of a block's 64 value columns."""

import pytest
import torch

from test_delta_chunks_gpu import exact, off, problem, run

from freetoken_b200.kernels import ops
from freetoken_b200.parts.delta import chunks_pay

gpu = pytest.mark.gpu
EDGES = [(63, 63), (64, 80), (65, 65), (127, 300), (128, 128), (129, 129)]


@gpu
@pytest.mark.parametrize("H,G,D,Dv", [(48, 8, 128, 80), (24, 24, 64, 128), (14, 2, 128, 16)])
@pytest.mark.parametrize("lens", [EDGES, [(1, 1)] + EDGES[2:3]])
def test_pairs_against_the_recurrence(H, G, D, Dv, lens):
    p = problem(lens, H, G, D, Dv, seed=H)
    want, want_state = exact(p)
    (out, state), (out1, state1) = run(p, True), run(p, False)
    for got, plain, w in ((out, out1, want), (state, state1, want_state)):
        assert off(got, w) < 1e-6  # (a few dozen 32-bit roundings of 2^-24 to a state that decays)
        assert off(got, w) <= max(1.1 * off(plain, w), 1e-7)
    torch.testing.assert_close(out.double(), want, rtol=1e-4, atol=2e-5)


@gpu
@pytest.mark.parametrize("what", ["q", "k", "v", "a", "b"])
@pytest.mark.parametrize("at,value", [(0, float("nan")), (40, float("inf")), (63, float("nan")), (70, float("-inf"))])
def test_no_number_reaches_no_earlier_token_in_blocks_of_64(what, at, value):
    p = problem([(100, 120), (90, 90)], 48, 8, 128, 128, seed=at)
    clean, clean_state = run(p, True)
    bad = dict(p, **{what: p[what].clone()})
    bad[what][at, 3 if what in "ab" else slice(None, None, 2)] = value
    (out, _), (tokens, _) = run(bad, True), run(bad, False)
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[100:], clean[100:])
    assert torch.isfinite(out[torch.isfinite(tokens)]).all()
    assert ops.read_status() == 0


@pytest.mark.parametrize("lens,heads,kv,dim,vdim,tokens_us,chunks_us", [
    ([80], 48, 8, 128, 128, 43, 40), ([96], 16, 4, 64, 64, 33, 29), ([128] * 8, 16, 4, 128, 128, 86, 56), ([256] * 4, 32, 4, 128, 128, 162, 75),
    ([512] * 8, 32, 8, 64, 64, 299, 161), ([128] * 16, 48, 48, 128, 64, 244, 198), ([80], 16, 4, 128, 32, 29, 32), ([128] * 16, 24, 3, 64, 16, 49, 77)])
def test_the_faster_kernel_is_named(lens, heads, kv, dim, vdim, tokens_us, chunks_us):
    assert chunks_pay(lens, False, heads, kv, dim, vdim) == (chunks_us < tokens_us)
