"""Infinities in the chunked recurrences: what the tensor core's pieces cannot carry comes out as 32-bit sums leave it."""

import pytest
import torch

import test_delta_chunks_gpu as delta

from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
INF = float("inf")


def kind(x):
    """0 for a number, 1 and -1 for infinities, 2 for NaN."""
    return torch.where(torch.isnan(x), 2, torch.isposinf(x).int() - torch.isneginf(x).int())


def copy_rows(x):
    """The same values in rows of the same stride."""
    return torch.empty(x.shape[0], x.stride(0), dtype=x.dtype, device=x.device)[:, : x.shape[1]].copy_(x)


@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 48), (6, 1, 64, 16), (48, 8, 128, 128), (40, 40, 64, 80)])
@pytest.mark.parametrize("what,at,value", [("v", 5, INF), ("v", 64, -INF), ("v", 98, 3.38e38), ("k", 33, INF), ("q", 20, -INF), ("b", 7, -INF),
                                           ("a", 70, INF), ("a", 9, -INF), ("state", 0, INF), ("state", 0, 3.4e38)])
def test_the_delta_rule_in_chunks_has_them_where_token_by_token_has_them(H, G, D, Dv, what, at, value):
    p = delta.problem([(99, 150), (70, 70), (130, 131)], H, G, D, Dv, seed=at + D)
    clean, _ = delta.run(p, True)
    bad = dict(p, **{what: p[what].clone() if what in ("a", "b", "state") else copy_rows(p[what])})
    if what == "state":
        bad["state"][p["slots"][0].item(), H // 2, 3, 11] = value
    else:
        bad[what][at, 3] = value
    (out, state), (tokens, token_state) = delta.run(bad, True), delta.run(bad, False)
    assert torch.equal(kind(out), kind(tokens)) and torch.equal(kind(state), kind(token_state))
    first = 0 if what == "state" else at
    assert torch.equal(out[:first], clean[:first]) and torch.equal(out[99:], clean[99:])
    rest = torch.isfinite(tokens)
    torch.testing.assert_close(out[rest], tokens[rest], rtol=1e-4, atol=2e-5)
    assert ops.read_status() == 0
