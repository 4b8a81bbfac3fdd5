"""Products in 32 bits on the tensor cores: at the edges of their tiles, and where :func:`ops.linear` hands over to them."""

import pytest
import torch

from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,N,K", [(1, 4, 4), (127, 129, 60), (128, 128, 64), (129, 1, 68), (300, 257, 1000)])
def test_against_64_bits(T, N, K):
    g = torch.Generator(device=DEV).manual_seed(T)
    x, w = torch.randn(T, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g)
    out = torch.full((T, N), float("nan"), device=DEV)
    ops.linear_split(x, w, out)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # chains of four products cut off four times, 2^-23 of at most their terms' sizes each; every 64 terms are added, rounded to 2^-24
    assert ((out - want).abs() <= (2.0 ** -21 + (K // 64 + 4) * 2.0 ** -24) * size).all()


def test_where_the_library_hands_over():
    for T, N, K, split in ((47, 16384, 64, False), (48, 12500, 64, True), (1000, 599, 64, False), (1000, 600, 64, True), (1000, 600, 66, False)):
        x, w, out = torch.randn(T, K, device=DEV), torch.randn(N, K, device=DEV), torch.empty(T, N, device=DEV)
        ops.variant_counts(reset=True)
        ops.linear(x, w, out)
        assert bool(ops.variant_counts().get("linear: float32 on the tensor cores")) == split
        torch.testing.assert_close(out.double(), x.double() @ w.double().T, rtol=1e-4, atol=1e-4)
    wide = torch.randn(1000, 128, device=DEV)  # rows that do not lie side by side stay with the library
    ops.variant_counts(reset=True)
    ops.linear(wide[:, :64], torch.randn(600, 64, device=DEV), torch.empty(1000, 600, device=DEV))
    assert not ops.variant_counts().get("linear: float32 on the tensor cores")


@pytest.mark.parametrize("small,large", [(2.0 ** -100, 2.0 ** 60), (2.0 ** -112, 2.0 ** 80), (2.0 ** -124, 2.0 ** 100)])
def test_numbers_that_the_third_piece_does_not_reach(small, large):
    """Three bfloat16 numbers hold a 32-bit one down to 2^-110; of smaller ones they leave out what lies under 2^-133."""
    g = torch.Generator(device=DEV).manual_seed(7)
    x, w = torch.randn(130, 256, device=DEV, generator=g) * small, torch.randn(130, 256, device=DEV, generator=g) * large
    out = torch.empty(130, 130, device=DEV)
    ops.linear_split(x, w, out)
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    left_out = 2.0 ** -134 * w.double().abs().sum(1)
    assert ((out - want).abs() <= (2.0 ** -21 + 8 * 2.0 ** -24) * size + left_out).all()
