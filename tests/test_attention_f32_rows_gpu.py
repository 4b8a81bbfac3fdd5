"""32-bit attention with several query rows a warp: bit for bit what a warp a row computes."""

import pytest
import torch

from test_pabavik_gpu import attention_problem

from freetoken_b200.engine.attention_plan import build_plan
from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(q, ks, vs, bt, seg, lens, Hkv, **kw):
    D, G = q.shape[2], q.shape[1] // Hkv
    plan = build_plan(lens, G, 16, None, Hkv, fixed_splits=1, sm_count=148)
    assert not plan.n_slots
    out = torch.full_like(q, float("nan"))
    ops.variant_counts(reset=True)
    ops.paged_attention(q, ks, vs, bt, seg, len(lens), torch.from_numpy(plan.items).to(DEV), plan.n_items, None, None, out, 16, 0.3 * D ** -0.5,
                        None, **kw)
    form = "up to %s rows a warp" % ("four" if D <= 64 and plan.n_items * Hkv > 148 else "two")
    assert [k for k in ops.variant_counts() if k.startswith("attention: float32")] == ["attention: float32, " + form]
    return out


@pytest.mark.parametrize("D", [16, 64, 80, 128, 256])
@pytest.mark.parametrize("Hq,Hkv,n,kv", [(6, 2, 70, 200), (4, 4, 33, 33), (16, 1, 9, 500), (8, 4, 700, 700)])
@pytest.mark.parametrize("tied,kw", [(False, {}), (True, {}), (False, dict(sink=0.5)), (False, dict(softcap=3.0))])
def test_rows_of_a_tile_are_rows_alone(D, Hq, Hkv, n, kv, tied, kw):
    """A prompt's tiles hold up to 16 rows, two or four a warp; its tokens as requests of their own have a row a warp (up to four or eight
    heads on a KV head), and few of them run with another number of warps (heads of 64)."""
    q, ks, vs, bt, seg = attention_problem(torch.float32, Hq, Hkv, D, 16, [(n, kv)], seed=D + n)
    vs = ks if tied else vs
    out = run(q, ks, vs, bt, seg, [(n, kv)], Hkv, **kw)
    alone = [(1, kv - n + i + 1) for i in range(n)]
    row = int(seg[0, 3])
    segs = torch.tensor([[i, 1, kv - n + i + 1, row] for i in range(n)], dtype=torch.int32, device=DEV)
    assert torch.equal(out, run(q, ks, vs, bt, segs, alone, Hkv, **kw))
    few = min(n, 3)
    last = segs[-few:] - torch.tensor([n - few, 0, 0, 0], dtype=torch.int32, device=DEV)
    assert torch.equal(out[-few:], run(q[-few:].contiguous(), ks, vs, bt, last, alone[-few:], Hkv, **kw))
    assert ops.read_status() == 0
