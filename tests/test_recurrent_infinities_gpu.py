"""Infinities in the chunked recurrences: what the tensor core's pieces cannot carry comes out as 32-bit sums leave it."""

import pytest
import torch

import test_delta_chunks_gpu as delta
import test_gla_chunks_gpu as gla

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


def gla_in_chunks(p, chunk):
    """Outputs and states in 64 bits as the chunk products have them: a value counts times a whole sum over the channels."""
    H, D, Dv = p["sizes"]
    q, k, v = (p[n].double().view(p["T"], -1, w) for n, w in (("q", D), ("k", D), ("v", Dv)))
    q = q * D ** -0.5
    if p["a_head"] is not None:
        logs = p["a_head"].double().log().expand(p["T"], H)[..., None].expand(-1, -1, D)
    else:
        logs = (torch.nn.functional.logsigmoid((p["z"] + p["bias"]).double()) / p["tau"]).view(-1, H, D)
    out, state = torch.empty(p["T"], H, Dv, dtype=torch.float64, device="cuda"), p["state"].double()
    for i, (q0, n, kv, _) in enumerate(p["info"].tolist()):
        slot = int(p["slots"][i])
        S = torch.zeros(H, D, Dv, dtype=torch.float64, device="cuda") if n == kv else state[slot].clone()
        for c0 in range(q0, q0 + n, chunk):
            rows = slice(c0, min(c0 + chunk, q0 + n))
            B = logs[rows].cumsum(0)
            for t in range(rows.stop - rows.start):
                w = (B[t] - B[: t + 1]).exp()  # [s, H, D]
                P = (q[rows][t] * k[rows][: t + 1] * w).sum(-1)
                out[c0 + t] = ((q[rows][t] * B[t].exp())[..., None] * S).sum(1) + (P[..., None] * v[rows][: t + 1]).sum(0)
            w = (B[-1] - B).exp()
            S = B[-1].exp()[..., None] * S + ((k[rows] * w)[..., None] * v[rows][:, :, None]).sum(0)
        state[slot] = S
    return out, state


@pytest.mark.parametrize("kw", [dict(D=128, Dv=128, chunk=64), dict(D=64, Dv=64, chunk=50), dict(D=64, Dv=96, chunk=64, decay="head"),
                                dict(D=128, Dv=72, chunk=64, decay="fixed")], ids=str)
@pytest.mark.parametrize("what,at,value", [("v", 5, INF), ("v", 100, -INF), ("v", 129, INF), ("k", 33, INF), ("k", 64, -INF), ("q", 20, INF),
                                           ("state", 0, -INF)])
def test_linear_attention_in_chunks_has_them_where_its_sums_have_them(kw, what, at, value):
    p = gla.problem([(130, 150), (70, 70)], H=2, bias=6.0, **kw)  # (no chunk's decay is zero in 32 bits)
    clean, _, taken = gla.run(p, kw["chunk"])
    bad = dict(p, **{what: p[what].clone() if what == "state" else copy_rows(p[what])})
    if what == "state":
        bad["state"][p["slots"][0].item(), 1, 11, 3] = value
    else:
        bad[what][at, 3] = value
    out, state, bad_taken = gla.run(bad, kw["chunk"])
    want, want_state = gla_in_chunks(bad, kw["chunk"])
    assert taken and bad_taken and not torch.isfinite(want).all()
    assert torch.equal(kind(out), kind(want)) and torch.equal(kind(state), kind(want_state))
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[130:], clean[130:])
    rest = torch.isfinite(want)
    torch.testing.assert_close(out[rest].double(), want[rest], rtol=1e-4, atol=2e-5)
    assert ops.read_status() == 0
