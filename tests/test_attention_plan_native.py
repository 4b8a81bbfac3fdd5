"""The native library's work lists (csrc/attention_plan.cu) against the plain statement of the same rules, number for number,
and that a step on a loaded library gets them: lists are made on the host before every step."""

import time

import pytest
import torch
from hypothesis import given, settings, strategies as st

from freetoken_b200.config.engine_config import EngineConfig
from freetoken_b200.config.spec import PartSpec
from freetoken_b200.engine import attention_plan
from freetoken_b200.engine.attention_plan import TC_ONE_TILE_COSTS, TC_TWO_TILE_COSTS, build_plan, plain_plan, tokens_per_tile
from freetoken_b200.engine.step import StepBuilder
from freetoken_b200.kernels import library
from freetoken_b200.parts import MIXERS, BuildEnv, Workspace

SEGMENT = st.tuples(st.sampled_from([1, 1, 1, 2, 5, 17, 33, 64, 300, 512, 1300, 2048, 4100]),
                    st.sampled_from([0, 0, 1, 3, 64, 500, 3000, 20000, 70000])).map(lambda qp: (qp[0], qp[0] + qp[1]))


def same(a, b):
    assert a.items.dtype == b.items.dtype and a.items.tolist() == b.items.tolist()
    assert (a.n_items, a.n_slots, a.tokens_per_tile, a.max_splits, a.est_us) == (b.n_items, b.n_slots, b.tokens_per_tile, b.max_splits, b.est_us)


@settings(max_examples=400, deadline=None)
@given(segs=st.lists(SEGMENT, min_size=0, max_size=40), group=st.sampled_from([1, 2, 3, 4, 6, 8, 16, 48]),
       tile=st.sampled_from([16, 64, 128, 256]), window=st.sampled_from([None, None, 1, 32, 500, 1024]), keep=st.sampled_from([0, 0, 4, 130]),
       n_kv=st.sampled_from([1, 2, 3, 8, 16, 48]), sm=st.sampled_from([1, 74, 148, 4096]), most=st.sampled_from([1, 32]),
       least=st.sampled_from([32, 256]), fixed=st.sampled_from([None, None, None, 0, 1, 2, 5, 16]), key_tile=st.sampled_from([0, 128]),
       costs=st.sampled_from([None, TC_ONE_TILE_COSTS, TC_TWO_TILE_COSTS]), sparse=st.sampled_from([None, None, None, (64, 16), (16, 3)]))
def test_native_lists_are_the_plain_ones(segs, group, tile, window, keep, n_kv, sm, most, least, fixed, key_tile, costs, sparse):
    lib = library.load()
    if sparse:
        window = None
    if fixed:  # (lists for graph replay: steps of single tokens and a few more)
        segs = [(min(q, 5), kv) for q, kv in segs if kv >= 5]
    elif tile // group < 8:
        segs = [(min(q, 300), kv) for q, kv in segs]
    args = (1 if sparse else tokens_per_tile(tile, group), tile, window, n_kv, sm, most, least, fixed, sparse, key_tile, costs, keep)
    native = attention_plan._native_plan(lib, segs, *args)
    same(native, plain_plan(segs, *args))


def test_a_list_longer_than_the_first_room():
    library.load()
    plan = build_plan([(8192, 8192)], 48, 64, None, 1)
    assert plan.n_items == 8192
    same(plan, plain_plan([(8192, 8192)], 1, 64, None, 1, 148, 32, 256, None, None, 0, None, 0))


def attention(heads, kv_heads, dim):
    env = BuildEnv(dtype=torch.bfloat16, device=torch.device("cpu"), max_seq_len=40000, max_step_tokens=8192,
                   workspace=Workspace(torch.device("cpu")))
    return MIXERS.build(PartSpec("gqa_attention", dict(hidden=1024, n_heads=heads, n_kv_heads=kv_heads, head_dim=dim, eps=1e-6,
                                                       position=PartSpec("none"), window=None)), env)


@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("segs", [[(2048, 2048)], [(512, 33280)] + [(1, 900 + 31 * i) for i in range(63)], [(512, 2048)] + [(1, 700)] * 8,
                                  [(1, 1000 + 50 * i) for i in range(64)]])
def test_a_step_does_not_wait_for_its_lists(monkeypatch, dim, segs):
    """Both forms compared, cuts searched, rows dealt: a fraction of what the plain statement takes (3 to 20 times as long)."""
    library.load()
    engine = type("E", (), dict(config=EngineConfig(model_path="", page_size=16)))
    part = attention(16, 4, dim)

    def once():
        builder = StepBuilder(engine, segs, fixed=all(q == 1 for q, _ in segs), sm_count=148)
        t = time.perf_counter()
        part.prepare(builder)
        return time.perf_counter() - t, builder

    native = min(once()[0] for _ in range(20))
    items = once()[1].sections
    monkeypatch.setattr(attention_plan.library, "loaded", lambda: None)
    plain = min(once()[0] for _ in range(20))
    for (_, a), (_, b) in zip(items, once()[1].sections):
        assert a.tolist() == b.tolist()
    assert native < 0.7 * plain, (native, plain)
