"""The gated delta rule in chunks against the recurrence in float64, beside the kernel that takes a
request's tokens one after the other."""

import pytest
import torch

from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
EPS = 1e-6


def problem(lens, H, G, D, Dv, seed=0, a_log=-1.0, same_keys=False):
    """lens: (tokens of this step, tokens after it) per request."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    T = sum(n for n, _ in lens)
    wide = rnd(T, 2 * G * D + H * Dv + 8).to(torch.bfloat16)
    if same_keys:
        wide[:, G * D:2 * G * D] = wide[:1, G * D:2 * G * D]
    info, q0 = [], 0
    for i, (n, kv) in enumerate(lens):
        info.append([q0, n, kv, i])
        q0 += n
    state = rnd(len(lens) + 2, H, Dv, D) * 0.3
    return dict(q=wide[:, :G * D], k=wide[:, G * D:2 * G * D], v=wide[:, 2 * G * D:2 * G * D + H * Dv], b=rnd(T, H).to(torch.bfloat16),
                a=rnd(T, H).to(torch.bfloat16), a_log=rnd(H) * 0.5 + a_log, dt_bias=rnd(H) - 1.0, state=state,
                slots=torch.randperm(len(lens) + 1, device=DEV, generator=g)[:len(lens)].to(torch.int32) + 1,
                info=torch.tensor(info, dtype=torch.int32, device=DEV), T=T, sizes=(H, G, D, Dv))


def run(p, chunks):
    H, G, D, Dv = p["sizes"]
    out = torch.full((p["T"], H, Dv), float("nan"), device=DEV)
    state = p["state"].clone()
    n = ops.delta_chunk_scratch(torch.bfloat16, p["T"], len(p["info"]), H, G, D, Dv)
    scratch = torch.full((n,), 255, dtype=torch.uint8, device=DEV) if chunks else None
    ops.variant_counts(reset=True)
    ops.delta_scan(p["q"], p["k"], p["v"], p["b"], p["a"], p["a_log"], p["dt_bias"], D ** -0.5, EPS, state, p["slots"], p["info"],
                   len(p["info"]), out, scratch=scratch)
    assert bool(ops.variant_counts().get("delta rule: chunks of 64 tokens, tcgen05")) == chunks
    return out, state


def exact(p):
    H, G, D, Dv = p["sizes"]
    f = lambda x: x.double()  # noqa: E731
    unit = lambda x: (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + EPS)).repeat_interleave(H // G, dim=1)  # noqa: E731
    q, k, v = unit(f(p["q"]).view(-1, G, D)) * D ** -0.5, unit(f(p["k"]).view(-1, G, D)), f(p["v"]).reshape(-1, H, Dv)
    beta = torch.sigmoid(f(p["b"]))
    g = torch.exp(-torch.exp(f(p["a_log"])) * torch.nn.functional.softplus(f(p["a"]) + f(p["dt_bias"]), threshold=1e9))
    out, state = torch.empty(p["T"], H, Dv, dtype=torch.float64, device=DEV), p["state"].double()
    for i, (q0, n, kv, _) in enumerate(p["info"].tolist()):
        slot = int(p["slots"][i])
        S = torch.zeros(H, Dv, D, dtype=torch.float64, device=DEV) if n == kv else state[slot].clone()
        for t in range(q0, q0 + n):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            out[t] = (S @ q[t][:, :, None])[..., 0]
        state[slot] = S
    return out, state


def off(x, want):
    return float((x.double() - want).norm() / want.norm())


MIXED = [(1, 1), (31, 31), (32, 40), (33, 33), (1, 9), (64, 100), (65, 65), (95, 95), (2, 2)]


@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 128), (6, 1, 64, 16), (3, 3, 64, 48), (8, 8, 128, 32), (16, 4, 64, 64), (2, 1, 128, 80)])
@pytest.mark.parametrize("lens,a_log,same", [(MIXED, -1.0, False), ([(300, 300)], -1.0, False), ([(129, 200), (40, 40)], 2.5, False),
                                             ([(200, 200)], -6.0, True)])
def test_chunks_against_the_recurrence(H, G, D, Dv, lens, a_log, same):
    """Ordinary decays, decays of e^-12 a token and of nearly one, and keys that are all the same."""
    p = problem(lens, H, G, D, Dv, seed=H + Dv, a_log=a_log, same_keys=same)
    want, want_state = exact(p)
    (out, state), (out1, state1) = run(p, True), run(p, False)
    # both add a few dozen 32-bit roundings of 2^-24 to a state that decays: 1e-6 with room; and the chunks lose nothing
    for got, plain, w in ((out, out1, want), (state, state1, want_state)):
        assert torch.isfinite(got).all()
        assert off(got, w) < 1e-6, (off(got, w), off(plain, w))
        # (keys that are all the same: every entry of the chunk's triangle counts, and is rounded: measured 1.18 to 1.24 times; all
        # others 0.6 to 1.02 times, or below two units of 2^-24)
        assert off(got, w) <= max((1.3 if same else 1.1) * off(plain, w), 1e-7), (off(got, w), off(plain, w))
    torch.testing.assert_close(out.double(), want, rtol=1e-4, atol=2e-5)
    untouched = [s for s in range(state.shape[0]) if s not in p["slots"].tolist()]
    assert torch.equal(state[untouched], p["state"][untouched])


@pytest.mark.parametrize("a_log", [-6.0, -1.0])
def test_a_long_prompt_loses_no_precision(a_log):
    p = problem([(2048, 2048)], 4, 2, 128, 64, seed=5, a_log=a_log)
    want, want_state = exact(p)
    (out, state), (out1, state1) = run(p, True), run(p, False)
    slots = p["slots"].tolist()
    state, state1, want_state = state[slots], state1[slots], want_state[slots]
    assert off(out, want) <= off(out1, want)
    assert off(state, want_state) <= off(state1, want_state)


def test_a_prompt_cut_anywhere():
    whole = problem([(200, 200)], 4, 2, 128, 32, seed=2)
    want, want_state = run(whole, True)
    for cuts in ((32, 168), (1, 199), (100, 100), (33, 31, 136)):
        state, at, outs = whole["state"].clone(), 0, []
        for n in cuts:
            part = {k: (v[at:at + n] if k in ("q", "k", "v", "b", "a") else v) for k, v in whole.items()}
            part.update(T=n, state=state, info=torch.tensor([[0, n, at + n, 0]], dtype=torch.int32, device=DEV))
            out, state = run(part, True)
            outs.append(out)
            at += n
        torch.testing.assert_close(torch.cat(outs), want, rtol=1e-5, atol=2e-6)
        torch.testing.assert_close(state, want_state, rtol=1e-5, atol=2e-6)


def test_what_is_not_taken_goes_token_by_token():
    assert ops.delta_chunk_scratch(torch.float32, 64, 1, 4, 2, 128, 64) == 0
    for H, G, D, Dv in ((4, 2, 96, 64), (4, 2, 128, 40), (4, 2, 256, 64)):
        assert ops.delta_chunk_scratch(torch.bfloat16, 64, 1, H, G, D, Dv) == 0
        assert ops._lib().ftk_delta_chunk_scratch(1, 64, 1, H, G, D, Dv) == 0
    for T, S in ((1, 1), (31, 1), (33, 2), (2048, 7)):
        assert ops.delta_chunk_scratch(torch.bfloat16, T, S, 4, 2, 128, 64) == ops._lib().ftk_delta_chunk_scratch(1, T, S, 4, 2, 128, 64)
    p = problem([(40, 40)], 4, 2, 128, 32)
    p["k"] = torch.cat([p["k"], p["k"][:, :4]], dim=1)[:, :256]  # rows of 260: no 16-byte copies
    out, _ = run(dict(p, k=p["k"].contiguous()), True)
    assert p["k"].stride(0) % 8
    scratch = torch.empty(ops.delta_chunk_scratch(torch.bfloat16, 40, 1, 4, 2, 128, 32), dtype=torch.uint8, device=DEV)
    got, state = torch.empty_like(out), p["state"].clone()
    ops.variant_counts(reset=True)
    ops.delta_scan(p["q"], p["k"], p["v"], p["b"], p["a"], p["a_log"], p["dt_bias"], 128 ** -0.5, EPS, state, p["slots"], p["info"], 1, got,
                   scratch=scratch)
    assert not ops.variant_counts().get("delta rule: chunks of 64 tokens, tcgen05")
    torch.testing.assert_close(got, out, rtol=1e-4, atol=2e-5)


def scan(p, out=None, eps=EPS, **kw):
    """One call with scratch for what is asked for; outputs start as NaN, scratch as 0xff."""
    H, G, D, Dv = p["sizes"]
    out = torch.full((p["T"], H, Dv), float("nan"), device=DEV) if out is None else out
    state = p["state"].clone()
    if kw:
        n = ops.delta_chunk_scratch(torch.bfloat16, p["T"], kw["n_long"], H, G, D, Dv)
        kw["scratch"] = torch.full((n,), 255, dtype=torch.uint8, device=DEV)
    ops.variant_counts(reset=True)
    ops.delta_scan(p["q"], p["k"], p["v"], p["b"], p["a"], p["a_log"], p["dt_bias"], D ** -0.5, eps, state, p["slots"], p["info"],
                   len(p["info"]), out, **kw)
    return out, state


@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 128), (6, 1, 64, 48)])
@pytest.mark.parametrize("lens", [[(1, 9), (64, 100), (5, 5), (1, 1), (96, 300), (63, 63), (2, 40)], [(200, 200)] + [(1, 30)] * 40,
                                  [(1, 30)] * 33 + [(64, 64)] + [(1, 5)] * 31 + [(70, 70)]])
def test_only_the_long_requests_of_a_step_go_in_chunks(H, G, D, Dv, lens):
    """A decoding request is the same, bit for bit, with and without a long neighbour: it stays token by token."""
    p = problem(lens, H, G, D, Dv, seed=D + len(lens))
    is_long = [n >= 64 for n, _ in lens]
    out, state = scan(p, long_from=64, n_long=sum(is_long))
    assert ops.variant_counts().get("delta rule: chunks of 64 tokens, tcgen05")
    (chunks, chunk_state), (tokens, token_state) = run(p, True), run(p, False)
    for i, (q0, n, _, _) in enumerate(p["info"].tolist()):
        slot, rows = int(p["slots"][i]), slice(q0, q0 + n)
        want, want_state = (chunks, chunk_state) if is_long[i] else (tokens, token_state)
        assert torch.equal(out[rows], want[rows]) and torch.equal(state[slot], want_state[slot]), (i, n)
    rest = [s for s in range(state.shape[0]) if s not in p["slots"].tolist()]
    assert torch.equal(state[rest], p["state"][rest])


def test_a_layer_takes_a_step_apart(monkeypatch):
    """The part hands over the number of its long requests, and no scratch where there is none."""
    from freetoken_b200.config.spec import PartSpec
    from freetoken_b200.parts import MIXERS, BuildEnv, Segment, StepState, Workspace
    from freetoken_b200.parts.delta import CHUNK_MIN_TOKENS

    calls = []
    real = ops.delta_scan
    monkeypatch.setattr(ops, "delta_scan", lambda *a, **kw: (calls.append({k: v for k, v in kw.items() if k != "scratch"}), real(*a, **kw)))
    env = BuildEnv(dtype=torch.bfloat16, device=torch.device(DEV), max_seq_len=512, max_step_tokens=512, workspace=Workspace(torch.device(DEV)))
    part = MIXERS.build(PartSpec("gated_delta", dict(hidden=64, n_heads=4, n_kv_heads=2, head_dim=64, v_head_dim=64, taps=1, eps=1e-6)), env)
    part.bind({n: torch.zeros(s.shape, device=DEV, dtype=torch.float32 if s.dtype == "float32" else torch.bfloat16)
               for n, s in part.param_specs().items()})
    for lens, n_long in (([1, CHUNK_MIN_TOKENS, 1, CHUNK_MIN_TOKENS - 1, 200], 2), ([1, 1, CHUNK_MIN_TOKENS - 1], 0)):
        info, q0 = [], 0
        for n in lens:
            info.append([q0, n, n, 0])
            q0 += n
        step = StepState(n_tokens=q0, segments=[Segment(i, a, n, kv) for i, (a, n, kv, _) in enumerate(info)], token_ids=None, positions=None,
                         seg_info=torch.tensor(info, dtype=torch.int32, device=DEV),
                         state_slots=torch.arange(len(lens), dtype=torch.int32, device=DEV), logit_rows=None, n_logit_rows=0,
                         attention_plans={}, decode_only=False)
        cache = type("C", (), dict(tensors={"s": torch.zeros(len(lens), 4, 64, 64, device=DEV)}))
        part.forward(torch.zeros(q0, 64, dtype=torch.bfloat16, device=DEV), step, cache, True)
        assert calls.pop() == (dict(long_from=CHUNK_MIN_TOKENS, n_long=n_long) if n_long else dict(z=None))


@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 48), (6, 1, 64, 16)])
@pytest.mark.parametrize("what", ["q", "k", "v", "a", "b"])
@pytest.mark.parametrize("at,value", [(0, float("nan")), (5, float("inf")), (17, float("nan")), (31, float("-inf")), (38, float("nan"))])
def test_a_value_that_is_no_number_reaches_no_earlier_token(H, G, D, Dv, what, at, value):
    """Nor another request, or a request's other outputs than those that the recurrence hands it to."""
    p = problem([(40, 50), (33, 33)], H, G, D, Dv, seed=at)
    clean, clean_state = run(p, True)
    bad = dict(p, **{what: p[what].clone()})
    bad[what][at, 3 if what in "ab" else slice(None, None, 2)] = value
    out, state = run(bad, True)
    tokens, token_state = run(bad, False)
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[40:], clean[40:])
    assert torch.equal(state[p["slots"][1]], clean_state[p["slots"][1]])
    # where the token-by-token kernel has numbers, there are numbers
    assert torch.isfinite(out[torch.isfinite(tokens)]).all()


@pytest.mark.parametrize("H,G,D,Dv", [(4, 2, 128, 48), (6, 1, 64, 16)])
@pytest.mark.parametrize("lens", [[(33, 33), (1, 7), (95, 200)], [(64, 64)]])
def test_unit_vectors_without_a_floor(H, G, D, Dv, lens):
    """unit_eps = 0, which vectors that are not zero allow: also where the last chunk is not full."""
    p = problem(lens, H, G, D, Dv, seed=3)
    (out, state), (plain, plain_state) = scan(p, eps=0.0, n_long=len(lens)), scan(p, eps=0.0)
    # (the same sums as with the usual floor of 1e-6 under squares of about D: the bound of the first test above)
    assert torch.isfinite(plain).all() and torch.isfinite(plain_state).all()
    torch.testing.assert_close(out, plain, rtol=1e-4, atol=2e-5)
    torch.testing.assert_close(state, plain_state, rtol=1e-4, atol=2e-5)


def test_requests_that_overlap_stay_within_scratch():
    """A table that names more chunks than the tokens allow: what scratch holds is worked on, the rest is left alone."""
    p = problem([(96, 96)] * 4, 4, 2, 128, 48)
    _, clean = run(p, True)
    p["info"][:, 0] = 0  # (four requests over the same 96 tokens of a step of 96: three chunks each, room for 96 / 32 + 4 = 7)
    p = {k: (v[:96] if k in ("q", "k", "v", "b", "a") else v) for k, v in p.items()}
    p["T"] = 96
    n = ops.delta_chunk_scratch(torch.bfloat16, 96, 4, 4, 2, 128, 48)
    guarded = torch.full((2 * n,), 171, dtype=torch.uint8, device=DEV)
    H, G, D, Dv = p["sizes"]
    out, state = torch.empty(96, H, Dv, device=DEV), p["state"].clone()
    ops.delta_scan(p["q"], p["k"], p["v"], p["b"], p["a"], p["a_log"], p["dt_bias"], D ** -0.5, EPS, state, p["slots"], p["info"], 4, out,
                   scratch=guarded)
    slots = p["slots"].long()
    assert torch.equal(state[slots[0]], clean[slots[0]]) and torch.equal(state[slots[1]], state[slots[0]])
    assert torch.equal(state[slots[2:]], p["state"][slots[2:]])  # (chunks 6 to 11: past the scratch)
    assert bool((guarded[n:] == 171).all())


def test_layers_of_different_sizes_share_a_workspace():
    """Each has scratch of its own from its first step on, with room for the largest: nothing that a step was given moves later."""
    from freetoken_b200.config.spec import PartSpec
    from freetoken_b200.parts import MIXERS, BuildEnv, Segment, StepState, Workspace

    env = BuildEnv(dtype=torch.bfloat16, device=torch.device(DEV), max_seq_len=512, max_step_tokens=480, workspace=Workspace(torch.device(DEV)),
                   max_decode_rows=2)
    layers = []
    for heads in (2, 6):
        part = MIXERS.build(PartSpec("gated_delta", dict(hidden=64, n_heads=heads, n_kv_heads=2, head_dim=64, v_head_dim=16, taps=1, eps=1e-6)), env)
        part.bind({n: torch.zeros(s.shape, device=DEV, dtype=torch.float32 if s.dtype == "float32" else torch.bfloat16)
                   for n, s in part.param_specs().items()})
        layers.append(part)

    def step(lens):
        info = [[sum(lens[:i]), n, n, 0] for i, n in enumerate(lens)]
        T = sum(lens)
        s = StepState(n_tokens=T, segments=[Segment(i, a, n, kv) for i, (a, n, kv, _) in enumerate(info)], token_ids=None, positions=None,
                      seg_info=torch.tensor(info, dtype=torch.int32, device=DEV), state_slots=torch.arange(len(lens), dtype=torch.int32, device=DEV),
                      logit_rows=None, n_logit_rows=0, attention_plans={}, decode_only=False)
        for part in layers:
            cache = type("C", (), dict(tensors={"s": torch.zeros(len(lens), part.n_heads, 16, 64, device=DEV)}))
            part.forward(torch.zeros(T, 64, dtype=torch.bfloat16, device=DEV), s, cache, True)
        return {k: b.data_ptr() for k, b in env.workspace._buffers.items() if k[0] == "delta.chunks"}

    first = step([200])
    assert len(first) == 2
    assert step([80] * 6) == first and step([480]) == first and step([81] * 5) == first  # (as many requests as fit in a step)
    assert sum(b.numel() for k, b in env.workspace._buffers.items() if k[0] == "delta.chunks") == sum(
        p.chunk_scratch(480, 6)[1] for p in layers)
