"""Latent query rows and head gates taken eight values at a time, beside the references and the forms for odd sizes."""

import pytest
import torch

import kernel_refs as ref
from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rnd(*shape, seed, dtype=torch.bfloat16):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("T,H,D,R,n_rot,inter,C,P,taken", [
    (11, 3, 16, 64, 64, False, 192, 256, True), (11, 3, 16, 64, 32, False, 64, 128, True), (7, 5, 8, 64, 64, True, 64, 144, True),
    (7, 5, 8, 16, 8, True, 24, 64, True), (300, 1, 128, 16, 0, False, 40, 64, True), (1, 1, 8, 16, 16, False, 8, 24, True),
    (9, 2, 16, 64, 8, False, 64, 128, False), (9, 2, 12, 64, 64, False, 64, 128, False), (9, 2, 16, 20, 16, True, 64, 128, False),
    (9, 2, 16, 64, 64, True, 60, 128, False)])
def test_latent_queries(T, H, D, R, n_rot, inter, C, P, taken):
    q, pos = rnd(T, H, D + R, seed=1), torch.randint(-3, 70, (T,), dtype=torch.int32, device=DEV, generator=torch.Generator(device=DEV).manual_seed(2))
    table = rnd(64, n_rot, seed=3, dtype=torch.float32) if n_rot else None
    got, want = torch.full((T, H, P), 3.0, dtype=q.dtype, device=DEV), torch.full((T, H, P), 3.0, dtype=q.dtype)
    ops.variant_counts(reset=True)
    ops.latent_query_rotate(q, D, R, n_rot, inter, pos, table, got, C)
    assert bool(ops.variant_counts().get("latent_query_rotate: eight values a thread")) == taken
    ref.latent_query_rotate(q.cpu(), D, R, n_rot, inter, pos.cpu().clamp(0, 63), table.cpu() if n_rot else None, want, C)
    torch.testing.assert_close(got.cpu().float(), want.float(), rtol=2.0 ** -7, atol=1e-6)  # one step of a bfloat16
    assert torch.equal(got[:, :, :C], torch.full_like(got[:, :, :C], 3.0)) and not bool(got[:, :, C + R:].any())


@pytest.mark.parametrize("T,H,D,taken", [(13, 6, 24, True), (1, 1, 8, True), (257, 3, 128, True), (13, 6, 20, False), (5, 2, 1, False)])
def test_head_gate(T, H, D, taken):
    wide, o = rnd(T, 50 + H, seed=1), rnd(T, H, D, seed=2)
    gate = 1.0 / (1.0 + torch.exp(-wide[:, 50:].float()))
    want = (o.float() * gate[:, :, None]).to(o.dtype)
    ops.variant_counts(reset=True)
    ops.head_gate(o, wide[:, 50:])
    assert bool(ops.variant_counts().get("head_gate: eight values a thread")) == taken
    torch.testing.assert_close(o.float(), want.float(), rtol=2.0 ** -7, atol=0.0)
    moved = rnd(T * H * D + 4, seed=2)[4:].view(T, H, D)  # (8 bytes into a 16-byte line)
    before = moved.clone()
    ops.head_gate(moved, wide[:, 50:])
    torch.testing.assert_close(moved.float(), (before.float() * gate[:, :, None]).to(o.dtype).float(), rtol=2.0 ** -7, atol=0.0)
