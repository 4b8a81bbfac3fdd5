"""The expert products on the CUDA cores (32-bit, and bfloat16 rows that the tensor-core kernels do not take) against float64,
at the edges of their tiles: rows an expert, columns, row lengths with and without 16-byte loads."""

import pytest
import torch

from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype,hidden,inter", [(torch.float32, 96, 68), (torch.float32, 131, 33), (torch.float32, 1024, 200),
                                                (torch.bfloat16, 100, 68), (torch.bfloat16, 77, 35)])
@pytest.mark.parametrize("rows", [[1, 0, 2, 4, 0, 3, 5, 8, 9, 0, 17, 1, 0, 0, 0, 0, 0, 0], [1], [0, 0, 7], [31, 0, 32, 33, 5], [64, 65, 0, 130, 40],
                                  [0] * 40 + [2] + [0] * 30 + [1]])
@pytest.mark.parametrize("act", ["silu", "swigluoai"])
def test_expert_products(dtype, hidden, inter, rows, act):
    g = torch.Generator(device=DEV).manual_seed(sum(rows) + hidden)
    E, R = len(rows), sum(rows)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    x = rnd(R, hidden).to(dtype)
    w1, w2 = (rnd(E, 2 * inter, hidden) * hidden ** -0.5).to(dtype), (rnd(E, hidden, inter) * inter ** -0.5).to(dtype)
    offsets = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32, device=DEV)
    routes = torch.randperm(R, device=DEV, generator=g).to(torch.int32)
    weights = torch.rand(R, device=DEV, generator=g)
    a, y = torch.full((R, inter), float("nan"), device=DEV, dtype=dtype), torch.full((R, hidden), float("nan"), device=DEV, dtype=dtype)
    ops.moe_gemm1_act(x, w1, offsets, act, 1.702, 7.0, a)
    ops.moe_gemm2(a, w2, offsets, routes, weights, y)
    e = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(rows, device=DEV))
    gu = torch.einsum("rk,rnk->rn", x.double(), w1.double()[e])
    gate, up = (t.to(dtype).double() for t in (gu[:, :inter], gu[:, inter:]))
    if act == "silu":
        want = gate * torch.sigmoid(gate) * up
    else:
        gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
        want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    # a 32-bit sum of n products in any order is within n 2^-24 of the sum of their sizes (about sqrt(n) here, for weights that
    # keep the spread of the rows); bfloat16 rounds gate, up and the result once each, 2^-9 of up to 16
    tol = dict(rtol=1e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(a.double(), want, **tol)
    down = torch.einsum("rk,rnk->rn", a.double(), w2.double()[e]) * weights.double()[routes.long()][:, None]
    torch.testing.assert_close(y.double(), down, **tol)


def test_more_experts_than_a_grid_has_tiles_of_few_rows():
    """44,000 experts of four rows: 66,000 tiles of eight rows do not fit a grid, 49,500 of 32 rows do."""
    E, K, I = 44000, 8, 4
    g = torch.Generator(device=DEV).manual_seed(1)
    x, w1 = torch.randn(4 * E, K, device=DEV, generator=g), torch.randn(E, 2 * I, K, device=DEV, generator=g)
    offsets = torch.arange(0, 4 * E + 1, 4, dtype=torch.int32, device=DEV)
    a = torch.full((4 * E, I), float("nan"), device=DEV)
    ops.moe_gemm1_act(x, w1, offsets, "silu", 1.702, 7.0, a)
    gu = torch.einsum("erk,enk->ern", x.view(E, 4, K).double(), w1.double()).view(4 * E, 2 * I)
    torch.testing.assert_close(a.double(), gu[:, :I] * torch.sigmoid(gu[:, :I]) * gu[:, I:], rtol=1e-5, atol=2e-5)  # (8 terms in 32 bits)
