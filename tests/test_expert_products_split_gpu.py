"""The 32-bit expert products on the tensor cores at the edges of their tiles (128 rows, 64 or 128 columns, 64 of k), and with
values that three bfloat16 numbers cannot hold."""

import pytest
import torch

from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def problem(hidden, inter, rows, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    E, R = len(rows), sum(rows)
    x = torch.randn(R, hidden, device=DEV, generator=g)
    w = torch.randn(E, 2 * inter, hidden, device=DEV, generator=g) * hidden ** -0.5
    w2 = torch.randn(E, hidden, inter, device=DEV, generator=g) * inter ** -0.5
    offsets = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32, device=DEV)
    return x, w, w2, offsets, torch.randperm(R, device=DEV, generator=g).to(torch.int32), torch.rand(R, device=DEV, generator=g)


def products(x, w, w2, offsets, routes, weights):
    a, y = torch.full((len(x), w2.shape[2]), float("nan"), device=DEV), torch.full_like(x, float("nan"))
    ops.variant_counts(reset=True)
    ops.moe_gemm1_act(x, w, offsets, "silu", 1.702, 7.0, a)
    ops.moe_gemm2(a, w2, offsets, routes, weights, y)
    assert ops.variant_counts() == {f"expert {which} product: float32 on the tensor cores": 1 for which in ("gate/up", "down")}
    assert ops.read_status() == 0
    return a, y


@pytest.mark.parametrize("hidden,inter", [(64, 64), (60, 68), (68, 60), (1024, 132), (4, 256)])
@pytest.mark.parametrize("rows", [[5], [127, 0, 128, 129], [0, 256, 1], [40] * 3])
def test_against_64_bits(hidden, inter, rows):
    p = problem(hidden, inter, rows, seed=hidden + len(rows))
    x, w, w2, offsets, routes, weights = p
    a, y = products(*p)
    e = torch.repeat_interleave(torch.arange(len(rows), device=DEV), torch.tensor(rows, device=DEV))
    for i in torch.unique(e):
        s = e == i
        xs, wi, w2i, r = x[s].double(), w[i].double(), w2[i].double(), weights[routes[s].long()].double()[:, None]
        gu, size = xs @ wi.T, xs.abs() @ wi.abs().T  # products, and the sums of their terms' sizes
        act, up = torch.nn.functional.silu(gu[:, :inter]), gu[:, inter:]
        down, down_size = (a[s].double() @ w2i.T) * r, (a[s].double().abs() @ w2i.abs().T) * r
        # A chain of four products cuts off four times, 2^-23 of at most its terms' sizes each; every 64 terms are then added, rounded
        # to 2^-24; what is left out is below that.  silu rises by 1.1 at most; it, its product and the route's weight add a few units.
        cut = lambda k: 2.0 ** -21 + (k // 64 + 4) * 2.0 ** -24  # noqa: E731
        bound = cut(hidden) * (1.1 * size[:, :inter] * up.abs() + size[:, inter:] * act.abs()) + 2.0 ** -21 * (act * up).abs()
        assert ((a[s] - act * up).abs() <= bound).all()
        assert ((y[s] - down).abs() <= cut(inter) * down_size + 2.0 ** -23 * down.abs()).all()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
def test_what_three_pieces_do_not_hold(value):
    """Such a value leaves every other row and column alone, and its own as sums of 32-bit numbers in order leave them."""
    x, w, w2, offsets, routes, weights = problem(132, 64, [70, 6])
    a, _ = products(x, w, w2, offsets, routes, weights)
    x = x.clone()
    x[3, 7] = value
    w[0, 5] = w[0, 64 + 5] = 0.0
    w[0, 5, 7] = w[0, 64 + 5, 7] = 1e-30
    got, _ = products(x, w, w2, offsets, routes, weights)
    rest = [i for i in range(76) if i != 3]
    cols = [j for j in range(64) if j != 5]
    assert torch.equal(got[rest][:, cols], a[rest][:, cols])
    gu = torch.tensor([float(x[3, 7]) * float(w[0, 5, 7])] * 2)  # (its other products there are zeros)
    want = torch.nn.functional.silu(gu[0]) * gu[1]
    torch.testing.assert_close(got[3, 5].cpu(), want, rtol=1e-5, atol=0.0, equal_nan=True)


def test_outputs_may_start_anywhere():
    """Rows and weights on 16-byte boundaries, outputs one element off: the same numbers, and nothing beside them."""
    x, w, w2, offsets, routes, weights = problem(128, 64, [70, 0, 6])
    a, y = products(x, w, w2, offsets, routes, weights)
    a1, y1 = (torch.full((t.numel() + 2,), 7.0, device=DEV) for t in (a, y))
    ops.moe_gemm1_act(x, w, offsets, "silu", 1.702, 7.0, a1[1:-1].view(a.shape))
    ops.moe_gemm2(a, w2, offsets, routes, weights, y1[1:-1].view(y.shape))
    for got, want in ((a1, a), (y1, y)):
        assert torch.equal(got[1:-1], want.view(-1)) and got[0] == got[-1] == 7.0
    assert ops.read_status() == 0
