"""Rotation with and without per-head norms: 16-byte and single-element forms, and the fused backward."""

import pytest
import torch

from slime_b200 import ops

pytestmark = pytest.mark.gpu


def _turn(x, pos, table, w, eps):
    d = x.shape[-1]
    if w is not None:
        x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w
    c, s = table[pos.long()][:, None, : d // 2], table[pos.long()][:, None, d // 2 :]
    lo, hi = x[..., : d // 2], x[..., d // 2 :]
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


@pytest.mark.parametrize("T,Hq,Hkv,D", [(1, 1, 1, 64), (3, 14, 2, 64), (77, 4, 4, 128), (1000, 32, 8, 128), (5, 3, 1, 256)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("pitch", [0, 8, 2])  # extra elements of a row: 2 leaves no 16-byte rows
def test_rotation_and_cache_write(kernels, T, Hq, Hkv, D, norm, pitch):
    """bf16 results of fp32 arithmetic: one rounding (2^-8) of values of at most sqrt(D)."""
    torch.manual_seed(T)
    row, eps = (Hq + 2 * Hkv) * D, 1e-6
    wide = torch.randn(T, row + pitch, device="cuda").bfloat16()
    qkv = wide[:, :row]
    pos = torch.randint(0, 50, (T,), device="cuda", dtype=torch.int32)
    table = ops.rope_cos_sin(64, D, 1e4, "cuda")
    qw, kw = ((torch.rand(D, device="cuda") + 0.5).bfloat16() if norm else None for _ in range(2))
    slots = torch.randperm(T + 3, device="cuda")[:T].to(torch.int32)
    slots[0] = -1
    x = qkv.reshape(T, -1, D).double()
    w64 = lambda w: None if w is None else w.double()  # noqa: E731
    q, k = _turn(x[:, :Hq], pos, table.double(), w64(qw), eps), _turn(x[:, Hq : Hq + Hkv], pos, table.double(), w64(kw), eps)
    kc, vc = (torch.zeros(T + 3, Hkv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    v = qkv.reshape(T, -1, D)[:, Hq + Hkv :].clone()
    rest = wide[:, row:].clone()
    ops.rope_kv_write(qkv, pos, table, slots, kc, vc, Hq, Hkv, D, qw, kw, eps)
    got = qkv.reshape(T, -1, D)
    torch.testing.assert_close(got[:, : Hq + Hkv].double(), torch.cat([q, k], 1), rtol=2**-8, atol=1e-4)
    assert torch.equal(got[:, Hq + Hkv :], v) and torch.equal(wide[:, row:], rest)
    held = slots >= 0
    assert torch.equal(kc[slots[held].long()], got[held, Hq : Hq + Hkv]) and torch.equal(vc[slots[held].long()], v[held])
    assert int(kc.abs().sum(-1).gt(0).any(-1).sum()) == T - 1


@pytest.mark.parametrize("T,Hq,Hkv,D", [(1, 1, 1, 64), (9, 14, 2, 64), (130, 8, 4, 128), (2000, 32, 8, 128)])
@pytest.mark.parametrize("shift", [0, 1])  # 1: norm weights that are not 16-byte aligned
def test_backward_of_norm_and_rotation(kernels, T, Hq, Hkv, D, shift):
    """Against 64 bits. Gradients of the rows: bf16 results (one rounding); of the weights: fp32 sums over T x heads terms of about one."""
    torch.manual_seed(T + D)
    eps, row = 1e-6, (Hq + 2 * Hkv) * D
    qkv, d = (torch.randn(T, row, device="cuda").bfloat16() for _ in range(2))
    pos = torch.randint(0, 50, (T,), device="cuda", dtype=torch.int32)
    table = ops.rope_cos_sin(64, D, 1e4, "cuda")
    qw, kw = ((torch.rand(D + shift, device="cuda") + 0.5).bfloat16()[shift:] for _ in range(2))
    x = qkv.double().view(T, -1, D)[:, : Hq + Hkv].clone().requires_grad_()
    w = [t.double().requires_grad_() for t in (qw, kw)]
    out = torch.cat([_turn(x[:, :Hq], pos, table.double(), w[0], eps), _turn(x[:, Hq:], pos, table.double(), w[1], eps)], 1)
    out.backward(d.double().view(T, -1, D)[:, : Hq + Hkv])
    v = d.view(T, -1, D)[:, Hq + Hkv :].clone()
    qw.main_grad = torch.ones(D, device="cuda")
    dqw, dkw = ops.rope_norm_bwd_(qkv, d, pos, table, qw, kw, Hq, Hkv, D, eps)
    got = d.view(T, -1, D)
    torch.testing.assert_close(got[:, : Hq + Hkv].double(), x.grad, rtol=2**-8, atol=2**-10)
    assert torch.equal(got[:, Hq + Hkv :], v) and dqw is None and qw.grad_added_to_main_grad
    tol = 1e-5 * (T * Hq) ** 0.5 + 1e-5
    torch.testing.assert_close(qw.main_grad.double() - 1, w[0].grad, rtol=1e-4, atol=tol)
    torch.testing.assert_close(dkw.double(), w[1].grad, rtol=2**-8, atol=tol)
