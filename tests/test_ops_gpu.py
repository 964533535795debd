"""Own training kernels against fp32 PyTorch references of the same op."""
import ctypes as C_

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def test_layernorm_fwd_bwd():
    from gcow_b200.ops import kernels as K
    torch.manual_seed(0)
    for rows, H in ((64, 1024), (1000, 768), (37, 128)):
        x = torch.randn(rows, H, device="cuda", requires_grad=True)
        g = (torch.rand(H, device="cuda") + 0.5).requires_grad_(True)
        b = torch.randn(H, device="cuda", requires_grad=True)
        y = K.layernorm(x, g, b, 1e-12)
        w = torch.randn(rows, H, device="cuda")
        (y.float() * w).sum().backward()
        gx, gg, gb = x.grad.clone(), g.grad.clone(), b.grad.clone()
        x.grad = g.grad = b.grad = None
        xr = x.detach().bfloat16().float().requires_grad_(True)
        yr = F.layer_norm(xr, (H,), g, b, 1e-12)
        (yr * w.bfloat16().float()).sum().backward()
        assert (y.float() - yr).abs().max().item() < 0.05
        assert (gx.float() - xr.grad).abs().max().item() < 0.05 * xr.grad.abs().max().item() + 1e-3
        assert (gg - g.grad).abs().max().item() < 0.02 * g.grad.abs().max().item() + 1e-2
        assert (gb - b.grad).abs().max().item() < 0.02 * b.grad.abs().max().item() + 1e-2


@pytest.mark.parametrize("H", [8, 248, 256, 264, 520, 776, 1024, 1032])
@pytest.mark.parametrize("rows", [1, 5, 4001, 13001])
def test_layernorm_rows_in_registers(H, rows):
    """Widths around each number of register chunks and the last one with any; fewer rows than warps and several per warp."""
    from gcow_b200.ops import kernels as K
    torch.manual_seed(H + rows)
    x = (torch.randn(rows, H, device="cuda") * 2 + 3).bfloat16()
    g, b = torch.randn(H, device="cuda"), torch.randn(H, device="cuda")
    y = K.layernorm(x, g, b, 1e-12)
    xd = x.double()
    r = (xd.var(1, unbiased=False, keepdim=True) + 1e-12).rsqrt()
    n = (xd - xd.mean(1, keepdim=True)) * r
    ref = n * g.double() + b.double()
    # bf16 rounds to 2^-9; the mean of H fp32 values of size up to 12 is off by less than 12 (H + 5) 2^-24, which counts once for
    # every value and once for the deviation
    bound = 2.0 ** -8 * ref.abs() + 12 * (H + 5) * 2.0 ** -24 * r * (1 + n.abs()) * g.double().abs() + 1e-6
    assert bool(((y.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("H", [8, 16, 24, 248, 256, 264, 520, 776, 1024, 1032])
@pytest.mark.parametrize("rows", [1, 5, 1280, 1281, 2400, 5003])
def test_layernorm_backward_with_a_row_ahead(H, rows):
    """Each number of column chunks, the narrowest rows, fewer rows than warps, both CTA sizes around the line between them and one to
    three rows a warp, against float64."""
    from gcow_b200.ops import kernels as K
    torch.manual_seed(H * 7 + rows)
    x = torch.randn(rows, H, device="cuda").bfloat16().requires_grad_(True)
    g, b = torch.randn(H, device="cuda", requires_grad=True), torch.randn(H, device="cuda", requires_grad=True)
    dy = torch.randn(rows, H, device="cuda").bfloat16()
    K.layernorm(x, g, b, 1e-12).backward(dy)
    xd, d, gd = x.detach().double(), dy.double(), g.detach().double()
    rs = (xd.var(1, unbiased=False, keepdim=True) + 1e-12).rsqrt()
    xh = (xd - xd.mean(1, keepdim=True)) * rs
    gg = d * gd
    dx = rs * (gg - gg.mean(1, keepdim=True) - xh * (gg * xh).mean(1, keepdim=True))
    # bf16 rounds to 2^-9. In fp32 the sums over H values, and the mean and deviation behind xh, are off by up to (H + 16) 2^-24 of the
    # sum of their terms' sizes (values of size up to 6, one more factor rs); the sums over the rows by up to rows * 2^-24 of theirs.
    eps = 8 * (H + 16) * 2.0 ** -24 * (1 + rs)
    size = rs * (gg.abs() + gg.abs().mean(1, keepdim=True) + (1 + xh.abs()) * (gg * xh).abs().mean(1, keepdim=True))
    assert bool(((x.grad.double() - dx).abs() <= 2.0 ** -8 * dx.abs() + eps * size + 1e-6).all())
    off = (eps + (rows + 64) * 2.0 ** -24) * d.abs() * (1 + xh.abs())
    assert bool(((g.grad.double() - (d * xh).sum(0)).abs() <= off.sum(0) + 1e-6).all())
    assert bool(((b.grad.double() - d.sum(0)).abs() <= off.sum(0) + 1e-6).all())


@pytest.mark.parametrize("rows", [5, 1281])
@pytest.mark.parametrize("H", [24, 1024])
def test_layernorm_backward_with_partial_sums_at_any_address(H, rows):
    """The partial sums of gamma's and beta's gradients at an address that is a multiple of 4 alone: the same bits, nothing beside them."""
    from gcow_b200 import _native
    lib, S = _native.cuda(), torch.cuda.current_stream().cuda_stream
    torch.manual_seed(H + rows)
    dy, x = (torch.randn(rows, H, device="cuda").bfloat16() for _ in range(2))
    gamma, mean, rstd = torch.randn(H, device="cuda"), x.float().mean(1), 1 / x.float().std(1)
    parts = lib.gcow_layernorm_bwd_parts(rows)
    got = []
    for off in (0, 1):
        part = torch.full((parts * 2 * H + 16,), 7.0, device="cuda")
        dx, dgb = torch.empty_like(x), torch.empty(2 * H, device="cuda")
        assert lib.gcow_layernorm_bwd(dy.data_ptr(), x.data_ptr(), gamma.data_ptr(), mean.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
                                      part[off:].data_ptr(), dgb.data_ptr(), rows, H, S) == 0
        assert bool((part[:off] == 7).all()) and bool((part[off + parts * 2 * H:] == 7).all())
        got.append((dx, dgb))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("parts,n,off", [(1, 262144, 0), (3, 262144, 0), (8, 262148, 0), (9, 262144, 0), (3, 262140, 0), (3, 262146, 0),
                                         (4, 300000, 1), (5, 1048579, 0), (70, 300, 0)])
def test_ordered_sums_of_whole_numbers(parts, n, off):
    """Both sides of every line between the three kernels: length, multiples of four, alignment, number of partials. Sums of whole
    numbers are exact."""
    from gcow_b200 import _native
    part = torch.randint(-1000, 1000, (parts * n + off,), device="cuda").float()[off:]
    out = torch.full((n + 8,), 7.0, device="cuda")
    rc = _native.cuda().gcow_reduce_partials(part.data_ptr(), out.data_ptr(), parts, n, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert torch.equal(out[:n], part.view(parts, n).sum(0)) and bool((out[n:] == 7).all())


def test_gelu_fwd_bwd():
    from gcow_b200.ops import kernels as K
    x = (torch.randn(4096, 1024, device="cuda") * 2).requires_grad_(True)
    y = K.gelu(x)
    y.float().sum().backward()
    xr = x.detach().bfloat16().float().requires_grad_(True)
    yr = F.gelu(xr)
    yr.sum().backward()
    assert (y.float() - yr).abs().max().item() < 0.02
    assert (x.grad - xr.grad).abs().max().item() < 0.02


def test_softmax_xent_loss_and_grad():
    from gcow_b200.ops import kernels as K
    torch.manual_seed(1)
    rows, V, ld = 300, 30522, 30528
    base = (torch.randn(rows, ld, device="cuda") * 3).bfloat16()
    src = base.clone().requires_grad_(True)
    logits = (src * 1.0)[:, :V]                      # non-leaf strided view, as the vocabulary GEMM returns
    target = torch.randint(0, V, (rows,), device="cuda")
    target[::7] = -100
    ref_in = base[:, :V].float().requires_grad_(True)
    ref = F.cross_entropy(ref_in, target, ignore_index=-100)
    ref.backward()
    loss = K.softmax_xent(logits, target, -100)
    loss.backward()
    assert abs(loss.item() - ref.item()) < 2e-3 * abs(ref.item())
    g = src.grad[:, :V].float()
    assert (g - ref_in.grad).abs().max().item() < 2e-2 * ref_in.grad.abs().max().item()
    assert float(src.grad[:, V:].abs().sum()) == 0.0


@pytest.mark.parametrize("rows", [1, 7, 255, 257, 4096, 4097])
@pytest.mark.parametrize("cols,ld", [(8, 8), (64, 64), (72, 80), (1000, 1000), (6144, 6144), (6152, 6152)])
def test_colsum_of_whole_numbers(rows, cols, ld):
    """The one-launch sum (up to 4096 rows of 6144 columns) and the two kernels behind it: whole numbers of at most 8, whose sums fp32 holds exactly."""
    from gcow_b200.ops import kernels as K
    g = torch.randint(-8, 9, (rows, ld), device="cuda").to(torch.bfloat16)[:, :cols]
    assert torch.equal(K.colsum(g), g.double().sum(0).float())


def test_colsum_and_preprocess():
    from gcow_b200.ops import kernels as K
    for rows, cols in ((5000, 1024), (16384, 1000), (777, 30), (129, 4096)):     # wide (16-byte) and narrow paths
        g = torch.randn(rows, cols, device="cuda").bfloat16()
        ref = g.float().sum(0)
        assert (K.colsum(g) - ref).abs().max().item() < 2e-3 * ref.abs().max().item() + 1e-2, (rows, cols)
    x = torch.randint(0, 256, (4, 32, 32, 3), dtype=torch.uint8, device="cuda")
    mean = [0.485 * 255, 0.456 * 255, 0.406 * 255]
    std = [0.229 * 255, 0.224 * 255, 0.225 * 255]
    y = K.u8_to_bf16_norm(x, mean, std)
    assert y.shape == (4, 3, 32, 32) and y.is_contiguous(memory_format=torch.channels_last)
    ref = (x.permute(0, 3, 1, 2).float() - torch.tensor(mean, device="cuda").view(1, 3, 1, 1)) / \
        torch.tensor(std, device="cuda").view(1, 3, 1, 1)
    assert (y.float() - ref).abs().max().item() < 0.02


def test_conv1x1_matches_torch():
    from gcow_b200.ops import kernels as K
    torch.manual_seed(2)
    x = torch.randn(8, 64, 28, 28, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_(True)
    w = (torch.randn(256, 64, 1, 1, device="cuda") * 0.1).requires_grad_(True)
    assert K.conv1x1_usable(x, w)
    y = K.conv1x1(x, w, None)
    y.float().square().mean().backward()
    gx, gw = x.grad.clone(), w.grad.clone()
    x.grad = w.grad = None
    yr = F.conv2d(x.float(), w)
    yr.square().mean().backward()
    assert y.shape == yr.shape and (y.float() - yr).abs().max().item() < 0.05 * yr.abs().max().item()
    assert (gx.float() - x.grad.float()).abs().max().item() < 0.05 * x.grad.float().abs().max().item() + 1e-6
    assert (gw - w.grad).abs().max().item() < 0.05 * w.grad.abs().max().item() + 1e-6


def test_linear_with_odd_vocabulary_width():
    from gcow_b200.ops import kernels as K
    torch.manual_seed(3)
    x = torch.randn(2, 64, 128, device="cuda", requires_grad=True)
    w = (torch.randn(1002, 128, device="cuda") * 0.05).requires_grad_(True)
    b = torch.zeros(1002, device="cuda", requires_grad=True)
    t = torch.randint(0, 1002, (128,), device="cuda")
    y = K.linear(x, w, b)
    assert y.shape == (2, 64, 1002)
    loss = K.softmax_xent(y.flatten(0, 1), t)
    loss.backward()
    gx, gw, gb = x.grad.clone(), w.grad.clone(), b.grad.clone()
    x.grad = w.grad = b.grad = None
    ref = F.cross_entropy(F.linear(x, w, b).flatten(0, 1), t)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 0.02
    for a, r in ((gx, x.grad), (gw, w.grad), (gb, b.grad)):
        assert (a.float() - r).abs().max().item() < 0.08 * r.abs().max().item() + 1e-5


def test_bert_tiny_own_vs_torch_ops():
    from gcow_b200.models import bert_tiny
    from gcow_b200 import ops
    torch.manual_seed(4)
    m = bert_tiny().cuda()
    ids = torch.randint(0, 1024, (4, 64), device="cuda")
    lab = torch.where(torch.rand(4, 64, device="cuda") < 0.15, ids, torch.full_like(ids, -100))
    nsp = torch.randint(0, 2, (4,), device="cuda")
    losses = {}
    grads = {}
    for be in ("torch", "own"):
        ops.set_backend(be)
        m.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = m(ids, None, lab, nsp)
        loss.backward()
        losses[be] = loss.item()
        grads[be] = m.layers[0].fc1.weight.grad.clone()
    ops.set_backend("own")
    assert abs(losses["own"] - losses["torch"]) < 0.05
    d = (grads["own"] - grads["torch"]).abs().max().item()
    assert d < 0.1 * grads["torch"].abs().max().item() + 1e-4


@pytest.mark.parametrize("C,hw,res,relu", [(64, 56, False, True), (256, 14, True, True), (2048, 7, True, True), (128, 28, False, False)])
def test_batchnorm_act_fused_matches_fp32_reference(C, hw, res, relu):
    """Fused BN(+add)(+ReLU) against the same computation done by PyTorch in fp32."""
    from gcow_b200.ops import nn as gnn, set_backend
    torch.manual_seed(C)
    N = 16
    mk = lambda: (torch.randn(N, C, hw, hw, device="cuda") * 2 + 0.5).bfloat16().contiguous(memory_format=torch.channels_last)
    x0, r0, w = mk(), mk(), mk()
    gamma, beta = torch.rand(C, device="cuda") + 0.5, torch.rand(C, device="cuda") - 0.5
    # reference: fp32 all the way
    ref_bn = torch.nn.BatchNorm2d(C).cuda()
    with torch.no_grad():
        ref_bn.weight.copy_(gamma); ref_bn.bias.copy_(beta)
    xr = x0.float().requires_grad_(True)
    rr = r0.float().requires_grad_(True) if res else None
    yr = ref_bn(xr)
    if res:
        yr = yr + rr
    if relu:
        yr = torch.relu(yr)
    (yr * w.float()).sum().backward()
    # own kernels
    set_backend("own")
    bn = gnn.BatchNorm2d(C).cuda()
    with torch.no_grad():
        bn.weight.copy_(gamma); bn.bias.copy_(beta)
    x = x0.clone().requires_grad_(True)
    r = r0.clone().requires_grad_(True) if res else None
    y = bn(x, residual=r, relu=relu)
    assert y.dtype == torch.bfloat16 and y.is_contiguous(memory_format=torch.channels_last)
    (y.float() * w.float()).sum().backward()
    tol = lambda ref: 0.012 * ref.abs().max().item() + 1e-2          # bf16 has 8 bits of mantissa
    assert (y.float() - yr).abs().max().item() < tol(yr)
    assert (x.grad.float() - xr.grad).abs().max().item() < tol(xr.grad)
    if res:
        assert (r.grad.float() - rr.grad).abs().max().item() < tol(rr.grad)
    assert (bn.weight.grad - ref_bn.weight.grad).abs().max().item() < 0.01 * ref_bn.weight.grad.abs().max().item() + 0.5
    assert (bn.bias.grad - ref_bn.bias.grad).abs().max().item() < 0.01 * ref_bn.bias.grad.abs().max().item() + 0.5
    assert (bn.running_mean - ref_bn.running_mean).abs().max().item() < 1e-3
    assert (bn.running_var - ref_bn.running_var).abs().max().item() < 1e-2
    # inference statistics
    bn.eval(); ref_bn.eval()
    ye = bn(x0, residual=r0 if res else None, relu=relu)
    yer = ref_bn(x0.float()) + (r0.float() if res else 0)
    yer = torch.relu(yer) if relu else yer
    assert (ye.float() - yer).abs().max().item() < tol(yer)


def test_pools_match_torch():
    from gcow_b200.ops import kernels as K
    torch.manual_seed(5)
    x = torch.relu(torch.randn(8, 64, 57, 57, device="cuda")).bfloat16().contiguous(memory_format=torch.channels_last)
    xa = x.clone().requires_grad_(True)
    xb = x.clone().float().requires_grad_(True)
    ya, yb = K.maxpool3x3s2(xa), F.max_pool2d(xb, 3, 2, 1)
    assert ya.shape == yb.shape and torch.equal(ya.float(), yb)
    w = torch.randn_like(yb)
    (ya.float() * w).sum().backward(); (yb * w).sum().backward()
    assert (xa.grad.float() - xb.grad).abs().max().item() < 0.02 * xb.grad.abs().max().item() + 1e-3
    xa2 = x.clone().requires_grad_(True); xb2 = x.clone().float().requires_grad_(True)
    pa, pb = K.global_avgpool(xa2), F.adaptive_avg_pool2d(xb2, 1)
    assert (pa.float() - pb).abs().max().item() < 0.01
    pa.float().sum().backward(); pb.sum().backward()
    assert (xa2.grad.float() - xb2.grad).abs().max().item() < 1e-5


def test_resnet_own_vs_torch_backends_agree():
    from gcow_b200.models import resnet18
    from gcow_b200 import ops
    torch.manual_seed(6)
    m = resnet18(num_classes=10).cuda().to(memory_format=torch.channels_last)
    x = torch.randn(8, 3, 64, 64, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    y = torch.randint(0, 10, (8,), device="cuda")
    res = {}
    for be in ("torch", "own"):
        ops.set_backend(be)
        m.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = F.cross_entropy(m(x).float(), y)
        loss.backward()
        res[be] = (loss.item(), m.conv1.weight.grad.clone())
    ops.set_backend("own")
    assert abs(res["own"][0] - res["torch"][0]) < 0.05
    d = (res["own"][1] - res["torch"][1]).abs().max().item()
    assert d < 0.15 * res["torch"][1].abs().max().item() + 1e-3


@pytest.mark.parametrize("k,stride,pad", [(3, 1, 1), (3, 2, 1), (1, 2, 0), (7, 2, 3)])
def test_conv_as_im2col_gemm_matches_torch(k, stride, pad):
    from gcow_b200.ops import kernels as K
    torch.manual_seed(k * 10 + stride)
    x = torch.randn(4, 16, 30, 30, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_(True)
    w = (torch.randn(24, 16, k, k, device="cuda") * 0.1).requires_grad_(True)
    b = torch.randn(24, device="cuda", requires_grad=True)
    y = K.conv_gemm(x, w, b, stride, pad)
    wgt = torch.randn_like(y.float())
    (y.float() * wgt).sum().backward()
    gx, gw, gb = x.grad.float().clone(), w.grad.clone(), b.grad.clone()
    x.grad = w.grad = b.grad = None
    xr = x.detach().float().requires_grad_(True)
    yr = F.conv2d(xr, w, b, stride=stride, padding=pad)
    (yr * wgt).sum().backward()
    tol = lambda r: 0.02 * r.abs().max().item() + 1e-2
    assert y.shape == yr.shape and (y.float() - yr).abs().max().item() < tol(yr)
    assert (gx - xr.grad).abs().max().item() < tol(xr.grad)
    assert (gw - w.grad).abs().max().item() < tol(w.grad)
    assert (gb - b.grad).abs().max().item() < tol(b.grad)


def test_batched_gemm_and_own_attention():
    from gcow_b200.ops import kernels as K
    torch.manual_seed(8)
    a = (torch.randn(6, 200, 72, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(6, 136, 72, device="cuda") * 0.5).bfloat16()
    ref = torch.einsum("bmk,bnk->bmn", a.float(), b.float())
    y = K.bmm_bf16(a, b, out_dtype=torch.float32)
    y2 = K.bmm_bf16(a.transpose(1, 2).contiguous(), b.transpose(1, 2).contiguous(), a_t=True, b_t=True, out_dtype=torch.float32)
    K.check_errors()
    assert (y - ref).abs().max().item() < 2e-2 and (y2 - ref).abs().max().item() < 2e-2
    # attention against scaled_dot_product_attention in fp32
    B, S, H, D = 2, 128, 4, 64
    qkv = (torch.randn(B, S, 3, H, D, device="cuda") * 0.7).bfloat16().requires_grad_(True)
    w = torch.randn(B, S, H * D, device="cuda")
    o = K.attention(qkv)
    (o.float() * w).sum().backward()
    K.check_errors()
    g = qkv.grad.float().clone()
    x = qkv.detach().float().requires_grad_(True)
    q, k, v = (x[:, :, i].transpose(1, 2) for i in range(3))
    oref = F.scaled_dot_product_attention(q, k, v).transpose(1, 2).reshape(B, S, H * D)
    (oref * w).sum().backward()
    assert (o.float() - oref).abs().max().item() < 0.03
    assert (g - x.grad).abs().max().item() < 0.05 * x.grad.abs().max().item() + 0.02


@pytest.mark.parametrize("shape", [(2, 128, 2, 64), (1, 256, 3, 64), (2, 384, 2, 64), (1, 512, 4, 64)])
def test_fused_attention_matches_fp32_reference(shape):
    """Forward and the three gradients of the fused tcgen05 attention against softmax(QK^T / sqrt d) V in fp32 on
    the same bf16-rounded inputs."""
    from gcow_b200.ops import kernels as K
    B, S, H, D = shape
    torch.manual_seed(sum(shape))
    qkv = (torch.randn(B, S, 3, H, D, device="cuda") * 0.8).bfloat16().requires_grad_(True)
    assert K.fused_attention_usable(qkv)
    w = torch.randn(B, S, H * D, device="cuda").bfloat16()
    o = K.fused_attention(qkv)
    (o.float() * w.float()).sum().backward()
    K.check_errors()
    g = qkv.grad.float().clone()
    x = qkv.detach().float().requires_grad_(True)
    q, k, v = (x[:, :, i].transpose(1, 2) for i in range(3))
    p = torch.softmax(q @ k.transpose(-1, -2) / D ** 0.5, dim=-1)
    oref = (p @ v).transpose(1, 2).reshape(B, S, H * D)
    (oref * w.float()).sum().backward()
    assert (o.float() - oref).abs().max().item() < 0.02
    for i, name in enumerate(("dq", "dk", "dv")):
        err = (g[:, :, i] - x.grad[:, :, i]).abs().max().item()
        assert err < 0.03 * x.grad[:, :, i].abs().max().item() + 0.01, (name, err)


def test_attention_module_routes_to_the_fused_kernel():
    from gcow_b200.ops import kernels as K, nn as gnn, set_backend
    set_backend("own")
    qkv = (torch.randn(1, 128, 3, 2, 64, device="cuda") * 0.5).bfloat16()
    before = K.launch_count()
    o = gnn.attention(qkv)
    assert K.launch_count() == before + 1 and o.shape == (1, 128, 128)      # one launch: the fused forward
    small = (torch.randn(1, 64, 3, 2, 64, device="cuda") * 0.5).bfloat16()  # 64 positions: the batched-GEMM path
    before = K.launch_count()
    gnn.attention(small)
    assert K.launch_count() == before + 3


def test_packed_sdpa_matches_plain_autograd(monkeypatch):
    from gcow_b200.ops import nn as gnn, set_backend
    torch.manual_seed(10)
    B, S, H, D = 2, 64, 4, 64
    base = (torch.randn(B, S, 3, H, D, device="cuda") * 0.5).bfloat16()
    w = torch.randn(B, S, H * D, device="cuda").bfloat16()
    outs = {}
    monkeypatch.setenv("GCOW_ATTENTION", "lib")          # the library arm of the own backend
    for be in ("torch", "own"):
        set_backend(be)
        qkv = base.clone().requires_grad_(True)
        o = gnn.attention(qkv * 1.0)
        (o * w).sum().backward()
        outs[be] = (o.detach().float(), qkv.grad.float())
    set_backend("own")
    assert (outs["own"][0] - outs["torch"][0]).abs().max().item() < 1e-2
    assert (outs["own"][1] - outs["torch"][1]).abs().max().item() < 2e-2 * outs["torch"][1].abs().max().item() + 1e-3


def test_fused_ffn_and_linear_residual_match_unfused():
    """x + fc2(gelu(fc1 x)) and r + lin(x) with every elementwise step inside GEMM epilogues, against fp32 PyTorch."""
    import torch.nn as nn
    import torch.nn.functional as F
    from gcow_b200.ops import nn as gnn, set_backend
    set_backend("own")
    torch.manual_seed(11)
    M, H, Fd = 512, 256, 1024
    fc1, fc2, proj = gnn.Linear(H, Fd).cuda(), gnn.Linear(Fd, H).cuda(), gnn.Linear(H, H).cuda()
    x0 = (torch.randn(4, M // 4, H, device="cuda") * 0.7).bfloat16()
    c0 = (torch.randn(4, M // 4, H, device="cuda") * 0.7).bfloat16()
    gy = (torch.randn(4, M // 4, H, device="cuda") * 0.5).bfloat16()

    def run(fused):
        for m in (fc1, fc2, proj):
            m.zero_grad(set_to_none=True)
        x, c = x0.clone().requires_grad_(True), c0.clone().requires_grad_(True)
        if fused:
            h = gnn.linear_residual(c, proj, x)
            y = gnn.ffn_residual(h, fc1, fc2)
        else:
            xf, cf = x.float(), c.float()
            h = xf + F.linear(cf, proj.weight, proj.bias)
            y = h + F.linear(F.gelu(F.linear(h, fc1.weight, fc1.bias)), fc2.weight, fc2.bias)
        y.backward(gy.to(y.dtype))
        return [y.detach().float(), x.grad.float(), c.grad.float()] + [p.grad.float().clone() for m in (fc1, fc2, proj) for p in m.parameters()]

    from gcow_b200.ops import kernels as K
    before = K.launch_count()
    got = run(True)
    assert K.launch_count() > before           # the fused functions ran, not the fallback
    K.check_errors()
    ref = run(False)
    for i, (a, b) in enumerate(zip(got, ref)):
        err = (a - b).abs().max().item() / (b.abs().max().item() + 1e-6)
        assert err < 3e-2, (i, err)


def test_fused_embeddings_match_pytorch():
    import torch.nn as nn
    from gcow_b200.ops import nn as gnn, set_backend
    torch.manual_seed(12)
    B, S, H, V = 4, 48, 256, 500
    tok, pos, typ = gnn.Embedding(V, H).cuda(), gnn.Embedding(64, H).cuda(), gnn.Embedding(2, H).cuda()
    ids = torch.randint(0, V, (B, S), device="cuda")
    ids[0, :10] = 7                                      # a long run of one id
    ty = torch.randint(0, 2, (B, S), device="cuda")
    gy = torch.randn(B, S, H, device="cuda").bfloat16()
    res = {}
    for be in ("torch", "own"):
        set_backend(be)
        for m in (tok, pos, typ):
            m.zero_grad(set_to_none=True)
        y = gnn.embed_sum3(ids, ty, tok, pos, typ)
        y.backward(gy.to(y.dtype))
        res[be] = [y.detach().float()] + [m.weight.grad.clone() for m in (tok, pos, typ)]
    set_backend("own")
    assert res["own"][0].dtype == torch.float32 and (res["own"][0] - res["torch"][0]).abs().max().item() < 2e-2
    for a, b in zip(res["own"][1:], res["torch"][1:]):
        assert (a - b).abs().max().item() < 1e-3 * max(1.0, b.abs().max().item())


def test_batchnorm_fork_adds_the_two_gradients_in_the_kernel():
    """bn(x, residual, relu, fork=True) returns two tensors on one memory; their gradients arrive separately and are
    added inside the backward kernel. Compared with fp32 PyTorch ops on the same values."""
    import torch.nn.functional as F
    from gcow_b200.ops import nn as gnn, set_backend
    set_backend("own")
    torch.manual_seed(13)
    N, C, H, W = 8, 64, 12, 12
    bn = gnn.BatchNorm2d(C).cuda()
    with torch.no_grad():
        bn.weight.uniform_(0.5, 1.5); bn.bias.uniform_(-0.3, 0.3)
    x0 = torch.randn(N, C, H, W, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    r0 = torch.randn(N, C, H, W, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    w1 = torch.randn(N, C, H, W, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    w2 = torch.randn(N, C, H, W, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    x, r = x0.clone().requires_grad_(True), r0.clone().requires_grad_(True)
    y1, y2 = bn(x, residual=r, relu=True, fork=True)
    assert y1.data_ptr() == y2.data_ptr() and y1 is not y2
    ((y1 * w1).sum() + (y2 * w2).sum()).backward()
    got = [y1.detach().float(), x.grad.float(), r.grad.float(), bn.weight.grad.clone(), bn.bias.grad.clone()]

    xf, rf = x0.float().requires_grad_(True), r0.float().requires_grad_(True)
    g, b = bn.weight.detach().clone().requires_grad_(True), bn.bias.detach().clone().requires_grad_(True)
    yr = F.relu(F.batch_norm(xf, None, None, g, b, True, 0.1, bn.eps) + rf)
    (yr * (w1.float() + w2.float())).sum().backward()
    ref = [yr.detach(), xf.grad, rf.grad, g.grad, b.grad]
    for i, (a, e) in enumerate(zip(got, ref)):
        err = (a - e).abs().max().item() / (e.abs().max().item() + 1e-6)
        assert err < 3e-2, (i, err)
    # only one of the two outputs used: the other gradient is absent
    bn.zero_grad(set_to_none=True)
    x = x0.clone().requires_grad_(True)
    y1, y2 = bn(x, relu=True, fork=True)
    (y2 * w2).sum().backward()
    xf = x0.float().requires_grad_(True)
    (F.relu(F.batch_norm(xf, None, None, bn.weight.detach(), bn.bias.detach(), True, 0.1, bn.eps)) * w2.float()).sum().backward()
    assert (x.grad.float() - xf.grad).abs().max().item() / xf.grad.abs().max().item() < 3e-2


@pytest.mark.parametrize("N,C,H,W", [(5, 8, 1, 1), (2, 64, 3, 5), (11, 2048, 17, 19), (1, 1024, 60, 37), (3, 256, 60, 59)])
@pytest.mark.parametrize("res,relu,fork", [(a, b, c) for a in (False, True) for b in (False, True) for c in (False, True)])
def test_batchnorm_every_form_of_the_sweeps(N, C, H, W, res, relu, fork):
    """Every combination of operands has its own kernels, each with several rows in flight: fewer rows than one CTA takes, fewer than the
    grid, just under and over 2, 3, 4 and 8 rows a thread. Against float64. A bf16 result is off by half a unit in its last place
    (2**-9 of it), a masked gradient that was written out carries the same into dx; the rest is fp32 sums."""
    from gcow_b200.ops import nn as gnn, set_backend
    set_backend("own")
    torch.manual_seed(C + H)
    mk = lambda: torch.randn(N, C, H, W, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    x0, r0, w1, w2 = mk(), mk(), mk(), mk()
    bn = gnn.BatchNorm2d(C).cuda()
    with torch.no_grad():
        bn.weight.uniform_(0.5, 1.5); bn.bias.uniform_(-0.3, 0.3)
    x, r = x0.clone().requires_grad_(True), (r0.clone().requires_grad_(True) if res else None)
    out = bn(x, residual=r, relu=relu, fork=fork)
    ys, ws = (list(out), [w1, w2]) if fork else ([out], [w1])
    torch.autograd.backward(ys, ws)

    col = lambda v: v.double().view(1, C, 1, 1)
    R, xd, ga = N * H * W, x0.double(), col(bn.weight.detach())
    mean, var = xd.mean((0, 2, 3), keepdim=True), xd.var((0, 2, 3), unbiased=False, keepdim=True)
    rstd = 1 / (var + bn.eps).sqrt()
    xh = (xd - mean) * rstd
    z = xh * ga + col(bn.bias.detach()) + (r0.double() if res else 0)
    y = ys[0].detach().double()
    want = z.clamp(min=0) if relu else z
    assert ((y - want).abs() <= 2**-8 * want.abs() + 1e-4).all()
    g = sum(w.double() for w in ws)
    if relu:
        g = torch.where(y > 0, g, torch.zeros_like(g))
    if res:
        assert ((r.grad.double() - g).abs() <= 2**-8 * g.abs()).all()
    db, dg = g.sum((0, 2, 3)), (g * xh).sum((0, 2, 3))
    assert ((bn.bias.grad.double() - db).abs() <= 1e-5 * g.abs().sum((0, 2, 3)) + 1e-5).all()
    assert ((bn.weight.grad.double() - dg).abs() <= 1e-5 * (g * xh).abs().sum((0, 2, 3)) + 1e-5).all()
    dx = ga * rstd * (g - col(db) / R - xh * col(dg) / R)
    assert ((x.grad.double() - dx).abs() <= 2**-8 * (dx.abs() + ga * rstd * g.abs()) + 1e-4 * ga * rstd).all()
    if not fork:                                             # inference: the same sweep, without a mask
        bn.eval()
        z = (xd - col(bn.running_mean)) / (col(bn.running_var) + bn.eps).sqrt() * ga + col(bn.bias.detach()) + (r0.double() if res else 0)
        want = z.clamp(min=0) if relu else z
        assert ((bn(x0, residual=r0 if res else None, relu=relu).double() - want).abs() <= 2**-8 * want.abs() + 1e-4).all()


@pytest.mark.parametrize("parts", [1, 2, 127, 129, 385, 443])
def test_batchnorm_sums_of_any_number_of_partials(parts):
    """The sums' second half takes 128 partials at a time, four times a turn: fewer, just more, just more than three, and nearly as many as the sweeps leave."""
    test_batchnorm_every_form_of_the_sweeps(1, 8, 1, parts * 256 - 3, False, True, False)     # 8 channels: 256 rows a partial


# Fewer rows than CTAs in a cluster, one CTA a cluster, clusters of 2 to 16, channels by 32 and by 16, shares of rows that differ by one, shares just
# within 52 KB and 104 KB (the lines themselves: test_batchnorm_forms_on_either_side_of_their_lines)
@pytest.mark.parametrize("N,C,H,W", [(1, 64, 1, 3), (1, 2048, 1, 1), (3, 2048, 7, 7), (17, 512, 7, 7), (13, 1024, 9, 11), (1, 128, 111, 113), (1, 128, 111, 121),
                                     (1, 256, 107, 61), (1, 64, 101, 259), (1, 2048, 61, 109), (1, 2048, 33, 50)])
@pytest.mark.parametrize("res,relu,fork", [(False, False, False), (False, True, False), (True, True, True), (True, False, False), (True, True, False), (False, True, True)])
def test_batchnorm_of_tensors_held_in_shared_memory(N, C, H, W, res, relu, fork):
    """Shapes that take the one-launch form, without other operands at least: against float64, and the running statistics."""
    from gcow_b200 import _native
    from gcow_b200.ops import nn as gnn
    R, lib = N * H * W, _native.cuda()
    lib.gcow_bn_launches.argtypes = [C_.c_int64, C_.c_int, C_.c_int, C_.c_int]
    assert lib.gcow_bn_launches(R, C, 0, 0) == 1
    test_batchnorm_every_form_of_the_sweeps(N, C, H, W, res, relu, fork)
    x = torch.randn(N, C, H, W, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    bn = gnn.BatchNorm2d(C).cuda()
    for _ in range(2):                                       # the second call finds the first one's sums in shared memory
        bn(x, residual=x if res else None, relu=relu)
    xd = x.double()
    mean, var = xd.mean((0, 2, 3)), xd.var((0, 2, 3), unbiased=R > 1)
    assert torch.allclose(bn.running_mean.double(), 0.19 * mean, rtol=1e-5, atol=1e-6)
    assert torch.allclose(bn.running_var.double(), 0.81 + 0.19 * var, rtol=1e-5, atol=1e-6)


# Per channel count the most rows that one launch takes: forward plain, with ReLU, with residual and ReLU, backward without and with another tensor
@pytest.mark.parametrize("C,lines", [(2048, (6656, 6656, 3328, 3328, 1664)), (1024, (13312, 13312, 6656, 6656, 3328)), (512, (13312, 13312, 9472, 6656, 5120)),
                                     (256, (13312, 13312, 11264, 13312, 6656)), (128, (26624, 20480, 11264, 13312, 10240)), (64, (26624, 26624, 18944, 13312, 10240)),
                                     (32, (0, 0, 0, 0, 0))])
def test_batchnorm_forms_on_either_side_of_their_lines(C, lines):
    """Which form a call takes and its results against float64, with the most rows that one launch takes and with one more. Values have a mean near 0 and a
    deviation near 1, so a result is off by bf16's rounding and a few fp32 roundings of numbers up to 5, and a sum by fp32's of its terms (below 2^-20 each)."""
    from gcow_b200 import _native
    from gcow_b200.ops import nn as gnn
    lib = _native.cuda()
    lib.gcow_bn_launches.argtypes = [C_.c_int64, C_.c_int, C_.c_int, C_.c_int]
    for (backward, extra), most in zip(((0, 0), (0, 2), (0, 3), (1, 0), (1, 3)), lines):
        for rows, launches in ((most, 1), (most + 1, 3)) if most else ((100, 3),):
            assert lib.gcow_bn_launches(rows, C, backward, extra) == launches, (backward, extra, rows)
            torch.manual_seed(rows)
            x, r, g = (torch.randn(1, C, rows, 1, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last) for _ in range(3))
            bn, x = gnn.BatchNorm2d(C, momentum=1.0).cuda(), x.requires_grad_(True)
            y = bn(x, residual=r.requires_grad_(True) if extra & 1 else None, relu=bool(extra & 2))
            y.backward(g)
            xd = x.detach().double()
            mean, var = xd.mean((0, 2, 3), keepdim=True), xd.var((0, 2, 3), unbiased=False, keepdim=True)
            xh = (xd - mean) / (var + bn.eps).sqrt()
            z = xh + (r.detach().double() if extra & 1 else 0)
            assert ((y.double() - (z.clamp(min=0) if extra & 2 else z)).abs() <= 2.0 ** -8 * z.abs() + 2.0 ** -18).all()
            gd = torch.where(y > 0, g, torch.zeros_like(g)).double() if extra & 2 else g.double()
            assert torch.allclose(bn.bias.grad.double(), gd.sum((0, 2, 3)), rtol=0, atol=2.0 ** -20 * rows)
            assert torch.allclose(bn.weight.grad.double(), (gd * xh).sum((0, 2, 3)), rtol=0, atol=2.0 ** -20 * rows)


@pytest.mark.parametrize("N,C,H,W", [(16, 2048, 7, 7), (1, 2048, 33, 50), (1, 128, 111, 113), (1, 64, 101, 259), (1, 256, 107, 61), (64, 512, 7, 7)])
@pytest.mark.parametrize("mean,low,high", [(10, 4, 15), (100, 64, 127)])
def test_batchnorm_variance_of_values_far_from_zero(N, C, H, W, mean, low, high):
    """The variance is what is left of two sums that are 100 and 10000 times as large. With these values, multiples of 2^-5 below 16 and of 2^-1 below 128, every fp32
    sum of 13 squares, a thread's share, is exact (less than 2^24 units), what lies behind in double is 2^-53 of 10000, and one rounding to fp32 is left."""
    from gcow_b200 import _native
    from gcow_b200.ops import nn as gnn
    lib = _native.cuda()
    lib.gcow_bn_launches.argtypes = [C_.c_int64, C_.c_int, C_.c_int, C_.c_int]
    assert lib.gcow_bn_launches(N * H * W, C, 0, 0) == 1
    torch.manual_seed(C + mean)
    x = (torch.randn(N, C, H, W, device="cuda") + mean).clamp(low, high).bfloat16().contiguous(memory_format=torch.channels_last)
    bn = gnn.BatchNorm2d(C, momentum=1.0).cuda()
    y = bn(x)
    xd = x.double()
    want, mu = xd.var((0, 2, 3)), xd.mean((0, 2, 3))
    assert ((bn.running_var.double() - want).abs() <= 2.0 ** -22 * want).all()
    assert ((bn.running_mean.double() - mu).abs() <= 2.0 ** -23 * mu).all()
    # x * scale + shift: two roundings of mean / deviation, and bf16's
    z = (xd - mu.view(1, C, 1, 1)) / (xd.var((0, 2, 3), unbiased=False) + bn.eps).sqrt().view(1, C, 1, 1)
    assert ((y.double() - z).abs() <= 2.0 ** -8 * z.abs() + 2.0 ** -21 * mean).all()


def test_batchnorm_counts_training_steps_lazily():
    """num_batches_tracked is counted on the host by the own path and lands in the tensor when the state is saved,
    when PyTorch's own path runs, and not twice."""
    from gcow_b200.ops import nn as gnn, set_backend
    set_backend("own")
    bn = gnn.BatchNorm2d(64).cuda()
    x = torch.randn(4, 64, 8, 8, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)
    for _ in range(5):
        bn(x, relu=True)
    assert int(bn.state_dict()["num_batches_tracked"]) == 5
    assert int(bn.state_dict()["num_batches_tracked"]) == 5
    set_backend("torch")
    bn(x.float())
    set_backend("own")
    assert int(bn.num_batches_tracked) == 6
