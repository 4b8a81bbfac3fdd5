"""Gated linear attention with chunks as matrix products against the recurrence in float64, beside the kernels that
take a chunk's tokens one after the other."""

import pytest
import torch

from freetoken_b200.kernels import ops
from freetoken_b200.parts.gla import chunk_list

pytestmark = pytest.mark.gpu
DEV = "cuda"
N_ROT = 32


def problem(lens, H, D, Dv, chunk, decay="channel", bias=2.0, tau=1.0, div=1, fac=False, rope=None, off=0, seed=0, dtype=torch.bfloat16):
    """lens: (tokens of this step, tokens after it) per request; decay: a decay per "channel", "head" or "fixed" head."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    T, Hq = sum(n for n, _ in lens), H // div
    wide = rnd(T, 2 * Hq * D + H * Dv + 16).to(dtype)[:, off:]
    info, q0 = [], 0
    for i, (n, kv) in enumerate(lens):
        info.append([q0, n, kv, i])
        q0 += n
    chunks, per_seg, single, multi = chunk_list(lens, chunk)
    pos = torch.arange(max(kv for _, kv in lens), device=DEV)[:, None] * 10000.0 ** (-torch.arange(N_ROT // 2, device=DEV) / (N_ROT // 2))
    a_head = None if decay == "channel" else torch.sigmoid(rnd(*((T, H) if decay == "head" else (H,))) + bias)
    return dict(q=wide[:, :Hq * D], k=wide[:, Hq * D:2 * Hq * D], v=wide[:, 2 * Hq * D:2 * Hq * D + H * Dv],
                z=rnd(T, H * D) if a_head is None else None, bias=rnd(H * D) + bias if a_head is None else None, tau=tau, a_head=a_head,
                k_fac=torch.rand(T, H, device=DEV, generator=g) if fac else None, rope=torch.cat([pos.cos(), pos.sin()], 1) if rope else None,
                neighbours=rope == "neighbours", state=rnd(len(lens) + 2, H, D, Dv) * 0.3, div=div,
                slots=torch.randperm(len(lens) + 1, device=DEV, generator=g)[:len(lens)].to(torch.int32) + 1,
                info=torch.tensor(info, dtype=torch.int32, device=DEV), chunks=torch.as_tensor(chunks, dtype=torch.int32, device=DEV),
                per_seg=torch.as_tensor(per_seg, dtype=torch.int32, device=DEV), single=single, multi=multi, T=T, sizes=(H, D, Dv))


def run(p, chunk):
    H, D, Dv = p["sizes"]
    n = p["chunks"].shape[0]
    out, state = torch.full((p["T"], H, Dv), float("nan"), device=DEV), p["state"].clone()
    ops.variant_counts(reset=True)
    ops.gla_scan(p["q"], p["k"], p["v"], None if p["z"] is None else p["z"].clone(), p["bias"], p["tau"], D ** -0.5, state, p["slots"],
                 p["info"], len(p["info"]), p["chunks"], n, p["per_seg"], p["single"], p["multi"],
                 torch.full((n, H, D, Dv), float("nan"), device=DEV), torch.full((n, H, D), float("nan"), device=DEV), out,
                 k_fac=p["k_fac"], a_head=p["a_head"], qk_div=p["div"], rope_table=p["rope"], neighbours=p["neighbours"], chunk=chunk)
    return out, state, bool(ops.variant_counts().get("gla_scan: chunks as products"))


def exact(p):
    H, D, Dv = p["sizes"]
    f = lambda x, w: x.double().view(p["T"], -1, w)  # noqa: E731
    q, k, v = f(p["q"], D) * D ** -0.5, f(p["k"], D), f(p["v"], Dv)
    if p["rope"] is not None:
        at = torch.cat([torch.arange(kv - n, kv, device=DEV) for _, n, kv, _ in p["info"].tolist()])
        c, s = p["rope"][at].double()[:, None].chunk(2, -1)
        half = N_ROT // 2
        for x in (q, k):
            i = (slice(0, N_ROT, 2), slice(1, N_ROT, 2)) if p["neighbours"] else (slice(0, half), slice(half, N_ROT))
            x0, x1 = x[..., i[0]].clone(), x[..., i[1]].clone()
            x[..., i[0]], x[..., i[1]] = x0 * c - x1 * s, x1 * c + x0 * s
    q, k = q.repeat_interleave(p["div"], 1), k.repeat_interleave(p["div"], 1)
    if p["k_fac"] is not None:
        k = k * p["k_fac"].double()[..., None]
    if p["a_head"] is not None:
        a = p["a_head"].double().expand(p["T"], H)[..., None].expand(-1, -1, D)
    else:
        a = torch.exp(torch.nn.functional.logsigmoid((p["z"] + p["bias"]).double()) / p["tau"]).view(-1, H, D)
    out, state = torch.empty(p["T"], H, Dv, dtype=torch.float64, device=DEV), p["state"].double()
    for i, (q0, n, kv, _) in enumerate(p["info"].tolist()):
        slot = int(p["slots"][i])
        S = torch.zeros(H, D, Dv, dtype=torch.float64, device=DEV) if n == kv else state[slot].clone()
        for t in range(q0, q0 + n):
            S = a[t][..., None] * S + k[t][..., None] * v[t][:, None]
            out[t] = (q[t][:, None] @ S)[:, 0]
        state[slot] = S
    return out, state


def rel(x, y):
    return float((x.double() - y).norm() / y.norm())


MIXED = [(129, 129), (1, 40), (300, 800), (20, 20), (64, 70), (65, 65), (191, 500)]  # several chunks beside single ones


@pytest.mark.parametrize("kw", [
    dict(lens=MIXED, H=3, D=128, Dv=128, chunk=64), dict(lens=MIXED, H=2, D=64, Dv=64, chunk=64), dict(lens=MIXED, H=2, D=128, Dv=64, chunk=32),
    dict(lens=MIXED, H=2, D=64, Dv=96, chunk=50), dict(lens=[(65, 65)], H=1, D=128, Dv=120, chunk=64), dict(lens=[(1000, 1000)], H=2, D=128, Dv=128, chunk=64),
    dict(lens=[(1000, 1100)], H=2, D=128, Dv=128, chunk=64, bias=-6.0), dict(lens=[(1000, 1100)], H=2, D=64, Dv=128, chunk=64, bias=8.0, tau=16.0),
    dict(lens=MIXED, H=4, D=128, Dv=64, chunk=64, decay="head", div=4, fac=True), dict(lens=MIXED, H=2, D=64, Dv=128, chunk=64, decay="fixed", rope="halves"),
    dict(lens=MIXED, H=2, D=128, Dv=128, chunk=64, decay="fixed", rope="neighbours", bias=4.0), dict(lens=MIXED, H=2, D=64, Dv=64, chunk=64, decay="head", bias=-8.0),
], ids=str)
def test_against_the_recurrence(kw):
    p = problem(**kw)
    want, want_state = exact(p)
    out, state, taken = run(p, kw["chunk"])
    plain, plain_state, other = run(p, 0)
    assert taken and not other
    # every path does 32-bit sums of at most D + 64 terms a chunk; decays are products of up to 64 factors: 2^-24 each, and
    # random signs leave a few units of it; both ways measure 0.3e-7 to 1.6e-7, and where decays are close to one the token-by-token
    # kernels 3.6e-6 and the products 3.0e-7
    used = p["slots"].long()
    for x, o, w in ((out, plain, want), (state[used], plain_state[used], want_state[used])):
        assert rel(x, w) <= max(2e-7, 1.1 * rel(o, w)), (rel(x, w), rel(o, w))
    rest = [s for s in range(state.shape[0]) if s not in used.tolist()]
    assert torch.equal(state[rest], p["state"][rest])


@pytest.mark.parametrize("kw", [dict(D=128, Dv=48, chunk=64), dict(D=128, Dv=136, chunk=64), dict(D=96, Dv=64, chunk=64), dict(D=64, Dv=68, chunk=64),
                                dict(D=64, Dv=64, chunk=16), dict(D=64, Dv=64, chunk=100), dict(D=64, Dv=64, chunk=64, off=1),
                                dict(D=64, Dv=64, chunk=64, dtype=torch.float32)], ids=str)
def test_what_stays_token_by_token(kw):
    p = problem([(300, 300)], H=2, **kw)
    out, state, taken = run(p, kw["chunk"])
    want, want_state = exact(p)
    assert not taken and rel(out, want) <= 1e-6 and rel(state[p["slots"].long()], want_state[p["slots"].long()]) <= 1e-6


@pytest.mark.parametrize("kw", [dict(D=128, Dv=128, chunk=64), dict(D=64, Dv=64, chunk=50), dict(D=64, Dv=96, chunk=64, decay="head", div=2)], ids=str)
@pytest.mark.parametrize("what", ["q", "k", "v", "decay"])
@pytest.mark.parametrize("at,value", [(0, float("nan")), (6, float("inf")), (21, float("nan")), (49, float("-inf")), (63, float("nan")), (129, float("nan"))])
def test_a_value_that_is_no_number_reaches_no_earlier_token(kw, what, at, value):
    """Nor another request: a later token counts for nothing, not for zero times what it holds."""
    p = problem([(130, 150), (70, 70)], H=2, **kw)
    clean, clean_state, taken = run(p, kw["chunk"])
    name = what if what != "decay" else "z" if p["a_head"] is None else "a_head"
    if name == "a_head" and value == value:
        value = float("nan")  # (a decay itself, not its logit)
    bad = dict(p, **{name: p[name].clone()})
    if name in ("q", "k", "v"):  # (their rows stay views of the same wide rows)
        cols = dict(q=p["q"], k=p["k"], v=p["v"])[name]
        bad[name] = torch.empty(cols.shape[0], cols.stride(0), dtype=cols.dtype, device=DEV)[:, : cols.shape[1]].copy_(cols)
    bad[name][at, ::2] = value
    out, state, bad_taken = run(bad, kw["chunk"])
    tokens, _, _ = run(bad, 0)
    assert taken and bad_taken
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[130:], clean[130:])
    assert torch.equal(state[p["slots"][1]], clean_state[p["slots"][1]])
    assert torch.isfinite(out[torch.isfinite(tokens)]).all()


@pytest.mark.parametrize("lens,chunk,kw,launches", [
    ([(130, 130), (1, 9)], 64, dict(D=64, Dv=64), 4), ([(130, 130)], 64, dict(D=64, Dv=64), 3), ([(1, 9)], 64, dict(D=64, Dv=64), 1),
    ([(130, 130), (1, 9)], 16, dict(D=64, Dv=64), 5), ([(130, 130)], 64, dict(D=64, Dv=64, decay="head"), 3),
    ([(130, 130)], 16, dict(D=64, Dv=64, decay="head"), 3)], ids=str)
def test_launches_are_counted(lens, chunk, kw, launches):
    """Single chunks one, products three, chunks side by side three and one for the decays of channels."""
    p = problem(lens, H=2, chunk=chunk, **kw)
    before = ops.launch_count()
    run(p, chunk)
    assert ops.launch_count() - before == launches
