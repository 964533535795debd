"""Epilogues of the CTA-pair GEMM and the fused attention against float64, at the edges of their tiles."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("M", [1024, 1025, 1100, 1279])
@pytest.mark.parametrize("N", [256, 288, 320])
def test_side_operands(M, N):
    """Residual, GELU with its argument kept, GELU' and GELU' + residual. Rows that end inside a warp's 32 and inside a
    tile, columns that end inside a warp's 128. One rounding to bf16 is at most 2^-9 of a value; the float32 sums are
    far below that."""
    from gcow_b200.ops import kernels as K
    torch.manual_seed(M + N)
    a = torch.randn(M, 512, device="cuda").bfloat16()
    w = (torch.randn(N, 512, device="cuda") / 16).bfloat16()
    bias = torch.randn(N, device="cuda")
    x = torch.randn(M, N, device="cuda").bfloat16() * 2
    p = a.double() @ w.double().T
    xd = x.double()
    cdf = 0.5 * (1 + torch.erf(xd / math.sqrt(2)))
    dgelu = cdf + xd * torch.exp(-xd * xd / 2) / math.sqrt(2 * math.pi)
    assert _rel(K.gemm_bf16(a, w, residual=x), p + xd) < 2 ** -9
    assert _rel(K.gemm_bf16(a, w, gelu_grad_of=x), p * dgelu) < 2 ** -9
    assert _rel(K.gemm_bf16(a, w, gelu_grad_of=x, residual=x), p * dgelu + xd) < 2 ** -9
    pre = torch.empty_like(x)
    y = K.gemm_bf16(a, w, bias=bias, gelu=True, pre_gelu_out=pre, residual=x)
    z = p + bias.double()
    assert _rel(pre, z) < 2 ** -9
    assert _rel(y, z * 0.5 * (1 + torch.erf(z / math.sqrt(2))) + xd) < 2 ** -9


def test_gelu_of_special_values():
    """0, both infinities, NaN and the underflow range of exp(-x^2 / 2), through an identity weight, one value per row."""
    from gcow_b200.ops import kernels as K
    v = torch.tensor([0.0, 20.0, -20.0, 13.2, -13.2, -14.0, 1e-30, -1e-30, 3e38, -3e38], device="cuda").bfloat16()
    x = torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    x[:v.numel(), 0] = v
    y = K.gemm_bf16(x, torch.eye(64, device="cuda", dtype=torch.bfloat16), gelu=True, out_dtype=torch.float32)[:v.numel(), 0].double()
    d = v.double()
    want = d * 0.5 * torch.erfc(-d / math.sqrt(2))
    # |Phi| is off by at most 1.5e-7 / 2, and by two roundings
    assert bool(((y - want).abs() <= d.abs() * 3e-7).all())
    x[0, 0] = float("nan")
    assert math.isnan(K.gemm_bf16(x, torch.eye(64, device="cuda", dtype=torch.bfloat16), gelu=True)[0, 0].item())


@pytest.mark.parametrize("B,S,H", [(74, 128, 1), (75, 128, 1), (37, 256, 1), (38, 256, 1), (37, 512, 1), (148, 128, 1), (149, 128, 1), (25, 256, 3), (25, 384, 2), (38, 512, 1)])
def test_attention_on_either_side_of_a_full_gpu(B, S, H):
    """As below, with 74 and 148 tiles, the most that have a CTA each in the backward and the forward kernels, and a few more."""
    test_attention(B, S, H)


@pytest.mark.parametrize("B,S,H", [(1, 128, 1), (2, 256, 3), (1, 384, 2), (3, 512, 4)])
def test_attention(B, S, H):
    """Forward and backward. Two roundings to bf16 on each path (P or dS, and the result): below 2^-8 of the norm."""
    from gcow_b200.ops import kernels as K
    torch.manual_seed(S)
    qkv = torch.randn(B, S, 3, H, 64, device="cuda").bfloat16().requires_grad_(True)
    o = K.fused_attention(qkv)
    go = torch.randn_like(o)
    o.backward(go)
    r = qkv.detach().double().requires_grad_(True)
    q, k, v = (r[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    ref = (torch.softmax(q @ k.transpose(-1, -2) / 8, -1) @ v).permute(0, 2, 1, 3).reshape(B, S, H * 64)
    ref.backward(go.double())
    assert _rel(o, ref.detach()) < 2 ** -8
    for i in range(3):
        assert _rel(qkv.grad[:, :, i], r.grad[:, :, i]) < 2 ** -8


@pytest.mark.parametrize("B,S,H", [(99, 128, 3), (331, 128, 1), (120, 384, 2), (80, 512, 2), (75, 256, 4), (148, 264, 6), (37, 384, 28)])
def test_attention_with_several_units_per_cta(B, S, H):
    """Two tiles per unit (of one head, of two heads, the last one alone, in long turns with pairs) and more units than SMs."""
    test_attention(B, S, H)


@pytest.mark.parametrize("B,S,H", [(1, 72, 1), (3, 120, 1), (150, 120, 1), (2, 136, 3), (80, 192, 2), (40, 200, 3), (5, 320, 2), (60, 384 - 8, 1),
                                   (70, 392, 2), (33, 504, 3)])
def test_attention_of_sequences_that_end_inside_a_tile(B, S, H):
    """Partial last blocks of keys and queries: of every kind of unit, an odd number of 64-row steps, a block of eight rows;
    and what lies behind the last sequence is not used."""
    from gcow_b200.ops import kernels as K
    test_attention(B, S, H)
    held = torch.full((B * S + 128, 3, H, 64), 7.0, device="cuda").bfloat16()
    qkv = held[:B * S].view(B, S, 3, H, 64)
    qkv.copy_(torch.randn(B, S, 3, H, 64, device="cuda"))
    held[B * S:] = float("nan")
    assert torch.isfinite(K.fused_attention(qkv)).all()


@pytest.mark.parametrize("S", [256, 512])
@pytest.mark.parametrize("order", [1, -1])
def test_attention_when_the_row_maximum_moves_between_key_blocks(S, order):
    """Keys that grow, or shrink, by a factor of four per 128 positions: the forward pass rescales at every block of keys, or
    never. Two roundings to bf16, as above."""
    from gcow_b200.ops import kernels as K
    torch.manual_seed(S)
    qkv = torch.randn(5, S, 3, 2, 64, device="cuda")
    grow = 4.0 ** (order * torch.arange(S // 128, device="cuda")).repeat_interleave(128)
    qkv[:, :, 1] *= grow.view(1, S, 1, 1)
    qkv = qkv.bfloat16().requires_grad_(True)
    o = K.fused_attention(qkv)
    go = torch.randn_like(o)
    o.backward(go)
    r = qkv.detach().double()
    q, k, v = (r[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    w = torch.softmax(q @ k.transpose(-1, -2) / 8, -1)
    assert _rel(o, (w @ v).permute(0, 2, 1, 3).reshape(5, S, 128)) < 2 ** -8
    dv = w.transpose(-1, -2) @ go.double().view(5, S, 2, 64).permute(0, 2, 1, 3)
    assert _rel(qkv.grad[:, :, 2], dv.permute(0, 2, 1, 3)) < 2 ** -8


@pytest.mark.parametrize("S", [72, 200, 376, 504])
def test_attention_of_rows_far_below_zero(S):
    """A shift of a row's scores does not change its softmax. A component that all keys have puts every scaled score near -150:
    against such a row's log-sum-exp, the zero score of a key that does not exist would be a probability beyond fp32."""
    from gcow_b200.ops import kernels as K
    torch.manual_seed(S)
    B, H = 3, 2
    qkv = torch.randn(B, S, 3, H, 64, device="cuda")
    qkv[:, :, 0, :, 0] = 40
    qkv[:, :, 1, :, 0] = -30
    qkv = qkv.bfloat16().requires_grad_(True)
    o = K.fused_attention(qkv)
    go = torch.randn_like(o)
    o.backward(go)
    K.check_errors()
    q, k, v = (qkv.detach().double()[:, :, i].permute(0, 2, 1, 3) for i in range(3))
    d = go.double().view(B, S, H, 64).permute(0, 2, 1, 3)
    p = torch.softmax(q @ k.transpose(-1, -2) / 8, -1)
    ref = p @ v
    ds = p * (d @ v.transpose(-1, -2) - (d * ref).sum(-1, keepdim=True)) / 8
    # P, dS and every result are rounded to bf16 (2^-9 each); so is the output, whose error comes into dS by way of delta
    e = ds.abs() + p * (d.abs() * ref.abs()).sum(-1, keepdim=True) / 8
    got = [o.detach().view(B, S, H, 64)] + [qkv.grad[:, :, i] for i in range(3)]
    want = [(ref, p @ v.abs()), (ds @ k, e @ k.abs()), (ds.transpose(-1, -2) @ q, e.transpose(-1, -2) @ q.abs()),
            (p.transpose(-1, -2) @ d, p.transpose(-1, -2) @ d.abs())]
    for x, (r, size) in zip(got, want):
        assert bool(((x.double().permute(0, 2, 1, 3) - r).abs() <= 2.0 ** -8 * (size + r.abs())).all())


@pytest.mark.parametrize("S", [72, 128])
def test_attention_of_tensors_at_odd_addresses(S):
    """Contiguous projections and gradients that do not start on 16 bytes are copied, not refused."""
    from gcow_b200.ops import nn as gnn
    torch.manual_seed(S)
    x = torch.randn(2, S, 3, 2, 64, device="cuda").bfloat16()
    go = torch.randn(2, S, 128, device="cuda").bfloat16()

    def run(qkv, g):
        qkv = qkv.requires_grad_(True)
        o = gnn.attention(qkv)
        o.backward(g)
        return o.detach(), qkv.grad

    def odd(t):
        return torch.cat((t.new_zeros(1), t.reshape(-1)))[1:].view(t.shape)
    for a, b in zip(run(x.clone(), go), run(odd(x), odd(go))):
        assert torch.equal(a, b)
