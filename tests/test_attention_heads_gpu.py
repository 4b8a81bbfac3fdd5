"""Heads of 64 and 256 on the tcgen05 attention kernels, and KV heads taken in several groups there, against the plain
statement of attention."""

import pytest
import torch

import kernel_refs as ref
from test_gizulorn_gpu import hide_the_passed
from test_pabavik_gpu import attention_problem, run_attention

from freetoken_b200.engine.attention_plan import build_plan
from freetoken_b200.kernels import ops
from freetoken_b200.parts.attention import attention_kernel_form
from freetoken_b200.parts.latent_attention import rows_filled, tile_split

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
# a probability is rounded to bfloat16 (2^-9 of itself; they add up to 1) and meets values of size up to 4: 8e-3, and the
# output is rounded once more (2^-9 of up to 4)
TOL = dict(rtol=2e-2, atol=1.5e-2)

MIXED = [(300, 300), (1, 1), (128, 128), (17, 273), (1, 130), (129, 257), (40, 40), (2, 64), (250, 1000), (1, 129)]


@pytest.mark.parametrize("D,tile", [(64, 128), (64, 256), (256, 128)])
@pytest.mark.parametrize("Hq,Hkv,P", [(12, 2, 16), (5, 5, 32), (7, 1, 64), (128, 1, 16), (3, 1, 48)])
def test_heads_of_64_and_256(D, tile, Hq, Hkv, P):
    assert ops.attention_tc_heads_fit(D, P, Hq // Hkv) and not ops.attention_tc_heads_fit(128, P, 1)
    for segs, kw in ((MIXED, {}), ([(140, 3000)], dict(force_split=True))):
        ops.variant_counts(reset=True)
        out, want, plan = run_attention(BF, Hq, Hkv, D, P, segs, tile, None, None, **kw)
        assert any(f"heads of {D}" in k for k in ops.variant_counts())
        torch.testing.assert_close(out.float(), want.float(), **TOL)
        assert bool(plan.n_slots) >= bool(kw)
    assert ops.read_status() == 0


@pytest.mark.parametrize("Hq,Hkv,P,splits", [(12, 2, 16, 1), (16, 1, 32, 3), (4, 4, 16, 5), (2, 1, 48, 16)])
def test_single_tokens_with_heads_of_64_in_the_form_for_few_rows(Hq, Hkv, P, splits):
    segs = [(1, 1), (1, 17), (1, 64), (1, 65), (1, 333), (1, 128), (1, 2000)]
    q, ks, vs, bt, seg = attention_problem(BF, Hq, Hkv, 64, P, segs)
    plan = build_plan(segs, Hq // Hkv, 16, None, Hkv, fixed_splits=splits, sm_count=74, key_tile=128)
    po = pm = None
    if plan.n_slots:
        po = torch.full((plan.n_slots, Hkv, 16, 64), float("nan"), device=DEV)
        pm = torch.full((plan.n_slots, Hkv, 16, 2), float("nan"), device=DEV)
    out, want = torch.full_like(q, float("nan")), torch.empty_like(q)
    ops.paged_attention(q, ks, vs, bt, seg, len(segs), torch.from_numpy(plan.items).to(DEV), plan.n_items, po, pm, out, 16, 0.1, None,
                        few_rows=True)
    ref.paged_attention(q, ks, vs, bt, seg, len(segs), None, 0, None, None, want, 16, 0.1, None)
    torch.testing.assert_close(out.float(), want.float(), **TOL)
    assert ops.read_status() == 0


@pytest.mark.parametrize("D,kv,splits,shape", [(128, 700, 5, (3, 40)), (64, 2000, 16, (1, 8)), (128, 5000, 8, (513, 1031)), (64, 100, 1, (64, 64))])
def test_a_weight_asked_for_ahead_changes_no_bit(D, kv, splits, shape):
    """Weights of less than a line, of no whole lines and of more than a line a thread; a step without split tiles."""
    q, ks, vs, bt, seg = attention_problem(BF, 12, 2, D, 16, [(1, kv)])
    plan = build_plan([(1, kv)], 6, 16, None, 2, fixed_splits=splits, sm_count=74, key_tile=128)
    po = pm = None
    if plan.n_slots:
        po, pm = torch.empty(plan.n_slots, 2, 16, D, device=DEV), torch.empty(plan.n_slots, 2, 16, 2, device=DEV)
    outs = []
    for ahead in (None, torch.ones(shape, dtype=BF, device=DEV)):
        outs.append(torch.full_like(q, float("nan")))
        ops.paged_attention(q, ks, vs, bt, seg, 1, torch.from_numpy(plan.items).to(DEV), plan.n_items, po, pm, outs[-1], 16, 0.1, None,
                            few_rows=True, ahead=ahead)
    assert torch.equal(outs[0], outs[1]) and bool(plan.n_slots) == (splits > 1)
    assert ops.read_status() == 0


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("Hq,Hkv,P,window,keep,split", [(6, 1, 16, 72, 0, 1), (48, 1, 16, None, 0, 3), (48, 1, 32, 200, 0, 3),
                                                        (256, 1, 16, 300, 0, 8), (8, 2, 48, 37, 5, 2), (128, 1, 16, 128, 129, 1)])
@pytest.mark.parametrize("tied", [True, False])
def test_windows_sinks_one_slab_and_split_heads(D, Hq, Hkv, P, window, keep, split, tied):
    """Values that are the keys (five 64-key steps in flight: pieces of every number of tiles) and values of their own; rows
    that a window has passed hold NaN."""
    sink = torch.randn(Hq, device=DEV, generator=torch.Generator(device=DEV).manual_seed(8)) * 1.5
    for segs, kw in (([(300, 300)], {}), ([(128, 128), (1, 40), (200, 517), (3, 3), (1, 1100)], {}), ([(256, 900)], dict(force_split=True)),
                     ([(1, 700), (1, 64), (1, 129), (1, 1500)], dict(fixed_splits=4))):
        problem = attention_problem(BF, Hq, Hkv, D, P, segs, seed=6)
        if window:
            problem = hide_the_passed(problem, window, keep, P)
        q, ks, vs, bt, seg = problem
        for s in (sink, None):
            out, want, _ = run_attention(BF, Hq, Hkv, D, P, segs, 128, window, s, problem=(q, ks, ks if tied else vs, bt, seg),
                                         kv_split=split, keep_first=keep, **kw)
            torch.testing.assert_close(out.float(), want.float(), **TOL)
    assert ops.read_status() == 0


def test_a_tile_of_equal_keys_and_one_far_larger_score():
    """Rows of 256: scores that grow by a thousand from tile to tile (the running maximum moves in each, and the output
    accumulator with it), and keys that are all alike (every weight the same)."""
    L, D = 1000, 256
    q, ks, vs, bt, seg = attention_problem(BF, 4, 1, D, 16, [(200, L)], seed=3)
    for rising in (True, False):
        flat = torch.ones(L, D, device=DEV) * ((torch.arange(L, device=DEV) // 128 * 4.0)[:, None] if rising else 1.0)
        for b in range(-(-L // 16)):
            n = min(16, L - 16 * b)
            ks[int(bt[1, b]), 0, :n] = flat[16 * b:16 * b + n].to(BF)
        qq = torch.ones_like(q)
        out, want, _ = run_attention(BF, 4, 1, D, 16, [(200, L)], 128, None, None, problem=(qq, ks, vs, bt, seg), scale=1.0)
        torch.testing.assert_close(out.float(), want.float(), **TOL)


def test_which_steps_go_there():
    """The rule over the forms that it accepts: heads of 64 wherever heads of 128 go, 256 in tiles of 128 rows; other sizes,
    other types, a bias or a cap as before."""
    for D in (16, 64, 80, 128, 256):
        for page in (8, 16, 24, 48):
            for group in (1, 6, 16, 48, 128, 130):
                for tokens, decode in ((1, True), (40, False), (128, False), (2000, False)):
                    plain = attention_kernel_form(BF, decode, group, tokens, D, page, None, 4096, plain_scores=True)
                    other = attention_kernel_form(BF, decode, group, tokens, D, page, None, 4096)
                    taken = page % 16 == 0 and group <= 128
                    if D == 64 and taken:
                        assert plain == attention_kernel_form(BF, decode, group, tokens, 128, page, None, 4096)
                    elif D == 256 and taken and (decode or tokens >= 128):
                        assert plain == (128, False)
                    else:
                        assert plain == other
                    if D != 128:
                        assert other[0] < 128 and not other[1]
    assert attention_kernel_form(torch.float32, False, 6, 2000, 256, 16, plain_scores=True) == (16, False)
    for heads in range(1, 257):
        s = tile_split(heads)
        assert heads % s == 0 and 1 <= heads // s <= 128 and rows_filled(heads, s) * 1.1 > max(
            rows_filled(heads, x) for x in range(1, heads + 1) if heads % x == 0)
