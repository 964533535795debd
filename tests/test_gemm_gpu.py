"""tcgen05 bf16 GEMM against an fp32 PyTorch reference of the same product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, bias=None, residual=None, gelu=False):
    y = a.float() @ b.float().t()
    if bias is not None:
        y = y + bias
    if gelu:
        y = torch.nn.functional.gelu(y)
    if residual is not None:
        y = y + residual.float()
    return y


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 256), (256, 512, 1024), (300, 520, 136),
                                   (4096, 1000, 2048), (77, 40, 72), (1024, 3072, 1024)])
def test_gemm_matches_fp32_reference(M, N, K):
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(M + N + K)
    a = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    ref = _ref(a, b)
    for dt in (torch.float32, torch.bfloat16):
        for rows in (128, 256):                      # both tile shapes
            y = K_.gemm_bf16(a, b, out_dtype=dt, tile_rows=rows)
            K_.check_errors()
            tol = 2e-2 if dt == torch.bfloat16 else 1e-3
            err = (y.float() - ref).abs().max().item() / (ref.abs().max().item() + 1e-6)
            assert err < tol, (dt, rows, err)


def test_gemm_epilogues():
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(0)
    M, N, K = 512, 768, 256
    a = (torch.randn(M, K, device="cuda") * 0.3).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.3).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N, device="cuda").bfloat16()
    ref = _ref(a, b, bias, res, True)
    for rows in (128, 256):
        y = K_.gemm_bf16(a, b, bias=bias, gelu=True, residual=res, tile_rows=rows)
        K_.check_errors()
        assert (y.float() - ref).abs().max().item() < 0.06
    acc = torch.ones(M, N, device="cuda")
    K_.gemm_bf16(a, b, out=acc, accumulate=True)
    assert (acc - (_ref(a, b) + 1)).abs().max().item() < 2e-2


def test_strided_operands_and_small_grid():
    from gcow_b200.ops import kernels as K_
    big = (torch.randn(640, 512, device="cuda") * 0.5).bfloat16()
    a = big[:, :256]                      # leading dimension 512, K 256
    b = (torch.randn(1024, 256, device="cuda") * 0.5).bfloat16()
    y = K_.gemm_bf16(a, b, out_dtype=torch.float32, max_ctas=3, tile_rows=256)   # several tiles per CTA
    K_.check_errors()
    assert (y - _ref(a, b)).abs().max().item() < 2e-2
    y = K_.gemm_bf16(a, b, out_dtype=torch.float32, max_ctas=3, tile_rows=128)
    K_.check_errors()
    assert (y - _ref(a, b)).abs().max().item() < 2e-2


def test_linear_autograd_matches_torch():
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(1)
    x = torch.randn(4, 64, 256, device="cuda", requires_grad=True)
    w = (torch.randn(384, 256, device="cuda") * 0.05).requires_grad_(True)
    b = torch.zeros(384, device="cuda", requires_grad=True)
    y = K_.linear(x, w, b)
    y.float().square().mean().backward()
    K_.check_errors()
    gx, gw, gb = x.grad.clone(), w.grad.clone(), b.grad.clone()
    x.grad = w.grad = b.grad = None
    yr = torch.nn.functional.linear(x, w, b)
    yr.square().mean().backward()
    assert (y.float() - yr).abs().max().item() < 0.05
    for g, r in ((gx, x.grad), (gw, w.grad), (gb, b.grad)):
        assert (g.float() - r).abs().max().item() <= 0.03 * r.abs().max().item() + 1e-6


@pytest.mark.parametrize("M,N,K", [(256, 512, 320), (304, 520, 136), (1024, 1024, 4096)])
def test_transposed_operands_without_copies(M, N, K):
    """dgrad (B stored [K,N]) and wgrad (both operands stored [K,rows]) layouts."""
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(7)
    a = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    ref = _ref(a, b)
    bt = b.t().contiguous()          # stored [K, N]
    at = a.t().contiguous()          # stored [K, M]
    scale = ref.abs().max().item()
    for rows in (128, 256):
        y1 = K_.gemm_bf16(a, bt, b_t=True, out_dtype=torch.float32, tile_rows=rows)
        y2 = K_.gemm_bf16(at, bt, a_t=True, b_t=True, out_dtype=torch.float32, tile_rows=rows)
        y3 = K_.gemm_bf16(at, b, a_t=True, out_dtype=torch.float32, tile_rows=rows)
        K_.check_errors()
        for y in (y1, y2, y3):
            assert (y - ref).abs().max().item() < 1e-3 * scale + 1e-3


def test_wgrad_split_k_matches_reference():
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(9)
    for M, N, K in ((8192, 256, 512), (16384, 1024, 1024), (4096, 64, 2304), (1000, 256, 256)):
        g = (torch.randn(M, N, device="cuda") * 0.3).bfloat16()
        x = (torch.randn(M, K, device="cuda") * 0.3).bfloat16()
        ref = g.float().t() @ x.float()
        y = K_.wgrad_gemm(g, x)
        K_.check_errors()
        assert y.shape == (N, K) and (y - ref).abs().max().item() < 2e-3 * ref.abs().max().item() + 1e-2


@pytest.mark.parametrize("M,N,K", [(1024, 256, 256), (1192, 320, 448), (1024, 1024, 1024), (5000, 1024, 256), (40000, 256, 320), (1 << 16, 256, 256)])
def test_wgrad_on_pairs_at_the_edges(M, N, K):
    """Tiles that overhang in both dimensions, rows that end inside a stage, one slice and many, a given result."""
    from gcow_b200 import _native
    from gcow_b200.ops import kernels as K_
    if _native.cuda().gcow_gemm2_wgrad_slices(N, K, M) <= 0:
        pytest.skip("clusters of two CTAs cannot be scheduled here")
    torch.manual_seed(M + N + K)
    # whole numbers up to 2: every sum of at most 65536 products is below 2^24, so fp32 holds it exactly in any order, and a row that
    # is lost or counted twice shows
    g, x = (torch.randint(-2, 3, (M, n), device="cuda").bfloat16() for n in (N, K))
    ref = g.double().t() @ x.double()
    out = torch.full((N, K), float("nan"), device="cuda")
    for y in (K_.wgrad_gemm(g, x), K_.wgrad_gemm(g, x, out)):
        K_.check_errors()
        assert y.shape == (N, K) and torch.equal(y.double(), ref)
    assert y.data_ptr() == out.data_ptr()


@pytest.mark.parametrize("M,N,K", [(1024, 256, 256), (1192, 320, 448), (1100, 256, 768), (5000, 1024, 1280), (40000, 256, 320), (2048, 512, 4096),
                                   (1500, 256, 8192), (1024, 256, 8448), (16384, 3072, 1024), (4096, 4096, 1024)])
def test_bias_gradient_beside_the_weight_gradient(M, N, K):
    """Column sums taken while the weight gradient's tiles pass: two tile columns, with a half of all rows to themselves each, up to more than a
    stage has groups of four rows for, an odd number of them, tiles that overhang, rows that end inside a stage, one slice, two accumulators, several; a single
    tile column, whose sums have a kernel of their own."""
    from gcow_b200 import _native
    from gcow_b200.ops import kernels as K_
    if _native.cuda().gcow_gemm2_wgrad_slices(N, K, M) <= 0:
        pytest.skip("clusters of two CTAs cannot be scheduled here")
    torch.manual_seed(M + N + K)
    # whole numbers, so that a sum below 2^24 is exact in any order
    g, x = (torch.randint(-2, 3, (M, n), device="cuda").bfloat16() for n in (N, K))
    w = torch.zeros(N, K, device="cuda", requires_grad=True)
    b = torch.zeros(N, device="cuda", requires_grad=True)
    for _ in range(2):                                      # results of the second pass do not depend on the first
        w.grad = b.grad = None
        K_.linear(x, w, b).backward(g)
        K_.check_errors()
        assert torch.equal(b.grad.double(), g.double().sum(0))
        assert torch.equal(w.grad.double(), g.double().t() @ x.double())


def test_bias_gradient_beside_weights_of_more_than_two_to_the_31_elements():
    """A single slice leaves no partial weight gradients to add up, so their number of elements is no limit; as sums of their own they may be
    as many as 4 (2^31 - 256). Whole numbers, exact in any order."""
    import ctypes
    from gcow_b200 import _native
    from gcow_b200.ops import kernels as K_
    M, N, K = 1024, 65536, 32768
    lib = _native.cuda()
    if lib.gcow_gemm2_wgrad_slices(N, K, M) != 1:
        pytest.skip("clusters of two CTAs cannot be scheduled here")
    torch.manual_seed(3)
    g, x = (torch.randint(-2, 3, (M, n), device="cuda").bfloat16() for n in (N, K))
    w = torch.zeros(N, K, device="cuda", requires_grad=True)
    b = torch.zeros(N, device="cuda", requires_grad=True)
    K_.linear(x, w, b).backward(g)
    K_.check_errors()
    assert torch.equal(b.grad.double(), g.double().sum(0))
    rows = [0, 1, 255, 256, 32767, N - 1]
    assert torch.equal(w.grad[rows].double(), g[:, rows].double().t() @ x.double())
    del w, b, g, x
    torch.cuda.empty_cache()
    n, p, i64 = 2 ** 31 + 4, ctypes.c_void_p, ctypes.c_int64
    part, out = torch.empty(2 * n, device="cuda"), torch.empty(n, device="cuda")
    ends = [0, 1, 2 ** 31 - 1, 2 ** 31, n - 1]
    part[ends] = torch.arange(1.0, 6.0, device="cuda")
    part[[n + e for e in ends]] = 10 * torch.arange(1.0, 6.0, device="cuda")
    bias_part, bias = torch.ones(3, 40, device="cuda"), torch.zeros(40, device="cuda")
    fn = lambda parts, n, at=0: lib.gcow_reduce_weight_bias(p(part.data_ptr() + at), p(out.data_ptr()), parts, i64(n), p(bias_part.data_ptr()), p(bias.data_ptr()), 3, 40,
                                                            p(torch.cuda.current_stream().cuda_stream))
    assert fn(2, n) == 0 and torch.equal(out[ends], 11 * torch.arange(1.0, 6.0, device="cuda")) and bool((bias == 3).all())
    bias.zero_()
    assert fn(0, 2 ** 40 + 1, 4) == 0 and bool((bias == 3).all())
    assert fn(2, 2 ** 33) == -1 and fn(2, 6) == -1 and fn(2, 8, 4) == -1 and fn(-1, 8) == -1
    del part, out
    torch.cuda.empty_cache()


def test_wgrad_slices_are_no_longer_than_slabs():
    """The tensor core's running sum loses a little at every step, so a slice of the rows on CTA pairs has no more stages of 128 than
    a slab of the one-CTA route, which doubles the slabs while the tiles fit 148 CTAs and 512 rows are left - twice as
    many where each pair has one item, whose two halves have an accumulator each."""
    from gcow_b200 import _native
    lib = _native.cuda()
    if lib.gcow_gemm2_wgrad_slices(256, 256, 1024) <= 0:
        pytest.skip("clusters of two CTAs cannot be scheduled here")
    for rows in (1024, 1088, 1152, 1192, 2048, 3000, 3136, 4096, 8192, 12544, 16384, 50176, 1 << 17):
        for n in (256, 320, 512, 768, 1024, 2304, 4096):
            for k in (256, 768, 1024, 2048, 3072, 4096):
                slabs = 1
                while (slabs < 64 and -(-n // 128) * -(-k // 256) * slabs * 2 <= 148 and rows % (2 * slabs) == 0
                       and rows // (2 * slabs) % 64 == 0 and rows // (2 * slabs) >= 512):
                    slabs *= 2
                slices, stages = lib.gcow_gemm2_wgrad_slices(n, k, rows), -(-rows // 128)
                items = -(-n // 256) * -(-k // 256) * slices
                run = -(-stages // slices)
                run = (run + 1) // 2 if items <= lib.gcow_gemm2_max_pairs() else run
                assert slices >= 1 and run <= -(-(rows // slabs) // 128), (rows, n, k)


@pytest.mark.parametrize("M,N,K", [(1024, 512, 256), (2048, 1024, 1024), (1100, 288, 192), (4096, 4096, 64)])
def test_pair_gemm_matches_fp32_reference(M, N, K, monkeypatch):
    """The CTA-pair kernel (cta_group::2) incl. ragged edges, a K that is not a whole stage, and every epilogue."""
    from gcow_b200 import _native
    from gcow_b200.ops import kernels as K_
    if not hasattr(_native.cuda(), "gcow_gemm2_bf16") or _native.cuda().gcow_gemm2_max_pairs() <= 0:
        pytest.skip("clusters of two CTAs cannot be scheduled here")
    monkeypatch.setattr(K_, "_pair_gemm", True)
    torch.manual_seed(M + N + K)
    a = (torch.randn(M, K, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(N, K, device="cuda") * 0.5).bfloat16()
    bias = torch.randn(N, device="cuda")
    res = torch.randn(M, N, device="cuda").bfloat16()
    before = K_.launch_count()
    y = K_.gemm_bf16(a, b)
    K_.check_errors()
    ref = _ref(a, b)
    assert (y.float() - ref).abs().max().item() / ref.abs().max().item() < 2e-2
    y = K_.gemm_bf16(a, b, bias=bias, residual=res)
    ref2 = _ref(a, b, bias=bias, residual=res)
    assert (y.float() - ref2).abs().max().item() / ref2.abs().max().item() < 2e-2
    pre = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    act = K_.gemm_bf16(a, b, bias=bias, gelu=True, pre_gelu_out=pre)
    K_.check_errors()
    ref_pre = _ref(a, b, bias=bias)
    assert (pre.float() - ref_pre).abs().max().item() / ref_pre.abs().max().item() < 2e-2
    ref_act = torch.nn.functional.gelu(ref_pre)
    assert (act.float() - ref_act).abs().max().item() / ref_act.abs().max().item() < 2e-2
    g = K_.gemm_bf16(a, b, gelu_grad_of=pre)
    x = pre.float()
    ref_g = ref * (0.5 * (1 + torch.erf(x / 2 ** 0.5)) + x * torch.exp(-0.5 * x * x) / (2 * 3.141592653589793) ** 0.5)
    assert (g.float() - ref_g).abs().max().item() / ref_g.abs().max().item() < 2e-2
    K_.check_errors()
    assert K_.launch_count() == before + 4
    if N % 64 == 0:        # B stored [K][N]: the data-gradient layout
        y = K_.gemm_bf16(a, b.t().contiguous(), b_t=True, residual=res)
        K_.check_errors()
        ref3 = _ref(a, b, residual=res)
        assert (y.float() - ref3).abs().max().item() / ref3.abs().max().item() < 2e-2


@pytest.mark.parametrize("M,N", [(1030, 264), (1300, 1288), (2305, 520), (260, 2600), (24, 48), (5000, 1000), (21000, 320), (26400, 26312), (26400, 26328)])
def test_every_tile_is_taken_once_in_either_order(M, N, monkeypatch):
    """Rows of tiles in groups of four and a shorter last group (more rows than columns), whole columns of tiles (fewer, or where only A
    with a column of the result fits the L2: both sides of that line), last rounds cut into halves, in all three kernels. The sums are whole numbers of at most 192,
    which bf16 and any order of addition hold exactly."""
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(M + N)
    a = torch.randint(-1, 2, (M, 192), device="cuda").bfloat16()
    b = torch.randint(-1, 2, (N, 192), device="cuda").bfloat16()
    ref = (a.float() @ b.float().t()).bfloat16()
    for rows in (0, 128, 256):
        assert torch.equal(K_.gemm_bf16(a, b, tile_rows=rows), ref), rows
    monkeypatch.setattr(K_, "_pair_gemm", True)
    assert torch.equal(K_.gemm_bf16(a, b), ref)
    K_.check_errors()


@pytest.mark.parametrize("M,N,K", [(2816, 2816, 2048), (3072, 3200, 2048), (5120, 5120, 4096), (5120, 5120, 4160), (4352, 4608, 4160), (4096, 4352, 4160),
                                   (2816, 2816, 8192), (4352, 4608, 8192)])
@pytest.mark.parametrize("b_t", [False, True])
def test_long_reductions_on_either_kernel(M, N, K, b_t):
    """Both sides of the lines between the pair and the one-CTA kernel for long plain reductions: a single round of tiles, as many rounds on
    either, finer ones on pairs, and their lengths. Sums of whole numbers are exact in fp32 and rounded once."""
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(M + K)
    a = torch.randint(-1, 2, (M, K), device="cuda").bfloat16()
    b = torch.randint(-1, 2, (K, N) if b_t else (N, K), device="cuda").bfloat16()
    bias = torch.randint(-9, 10, (N,), device="cuda").float()
    got = K_.gemm_bf16(a, b, bias=bias, b_t=b_t)
    assert torch.equal(got, K_.gemm_bf16(a, b, bias=bias, b_t=b_t, tile_rows=256))
    rows = slice(M // 2, M // 2 + 64)
    assert torch.equal(got[rows], (a[rows].double() @ (b if b_t else b.t()).double() + bias.double()).float().bfloat16())
    K_.check_errors()


# Both sides of the lines: rows of 64, 128 and 256 columns, 8, 24, 37, 74 and 148 tiles, 128 and 512 deep, a single low row, rows that are not whole vectors
@pytest.mark.parametrize("M,N,K", [(1, 256, 512), (7, 32, 64), (2048, 64, 64), (2300, 64, 64), (6144, 128, 128), (6145, 128, 128), (9472, 256, 128), (9473, 256, 64),
                                   (18944, 256, 64), (18945, 256, 64), (37900, 256, 192), (300, 1024, 768), (1000, 4096, 512), (2048, 2048, 768), (2048, 2048, 832),
                                   (300, 192, 72), (520, 96, 256)])
@pytest.mark.parametrize("b_t", [False, True])
def test_every_form_on_either_side_of_the_dispatch(M, N, K, b_t, monkeypatch):
    """The kernel that the rule takes against the one-CTA kernel: every epilogue, operands and results with rows apart, the result in the residual's
    place. Whole numbers, so the sums are exact and rounded once in both; GELU and GELU' have the same arithmetic in both."""
    from gcow_b200.ops import kernels as K_
    torch.manual_seed(M + N + K)
    mk = lambda r, c, lo, hi: torch.randint(lo, hi, (r, c + 8), device="cuda").bfloat16()[:, :c]      # rows apart
    a, b, res, x = mk(M, K, -1, 2), mk(K, N, -1, 2) if b_t else mk(N, K, -1, 2), mk(M, N, -8, 9), mk(M, N, -3, 4)
    bias, pre = torch.randint(-9, 10, (N,), device="cuda").float(), {}
    forms = [dict(), dict(bias=bias), dict(bias=bias, gelu=True), dict(residual=res), dict(bias=bias, residual=res)]
    if N % 32 == 0:
        forms += [dict(gelu_grad_of=x), dict(gelu_grad_of=x, residual=res), dict(bias=bias, gelu=True, pre_gelu_out=0), dict(gelu=True, residual=res, pre_gelu_out=0)]
    for form in forms:
        got = []
        for pair in (None, False):
            monkeypatch.setattr(K_, "_pair_gemm", pair)
            out, kw = mk(M, N, 0, 1), dict(form)
            if "pre_gelu_out" in kw:
                kw["pre_gelu_out"] = mk(M, N, 0, 1)
            K_.gemm_bf16(a, b, b_t=b_t, out=out, **kw)
            got.append((out, kw.get("pre_gelu_out")))
        assert torch.equal(got[0][0], got[1][0]), sorted(form)
        assert got[0][1] is None or torch.equal(got[0][1], got[1][1])
    K_.check_errors()


# Few rows of a wide result, on both sides of each line: 8, 16, 128 and 384 rows, 16, 37, 74 and 148 tiles, 64 K elements of A
@pytest.mark.parametrize("M,N,K", [(2, 4096, 512), (16, 4160, 512), (17, 4160, 512), (8, 6208, 64), (8, 9472, 192), (8, 9536, 64), (9, 9536, 64), (16, 9536, 1536), (40, 9536, 1536),
                                   (128, 19008, 64), (128, 38144, 2048), (129, 19008, 64), (256, 19008, 64), (300, 12288, 64), (300, 19008, 128), (300, 19008, 1024)])
def test_every_form_of_few_rows_on_either_side_of_the_dispatch(M, N, K, monkeypatch):
    test_every_form_on_either_side_of_the_dispatch(M, N, K, False, monkeypatch)


@pytest.mark.parametrize("M,N,K", [(8, 32, 64), (300, 96, 64), (1100, 1120, 192), (19000, 544, 64)])
@pytest.mark.parametrize("shift", [0, 1])
def test_pair_gemm_side_operands_with_everything(M, N, K, shift, monkeypatch):
    """A residual behind bias, kept argument and GELU; bias and residual around a GELU' factor; blocks and rows that do not exist; a bias that vectors
    cannot read; the result in the residual's place. Products, biases and residuals are whole numbers, so what is left is the approximation of
    Phi (1.5e-7 and a few 2^-24 of fp32 evaluation, times |argument| or |product|, at most K + 9) and bf16's rounding."""
    from gcow_b200.ops import kernels as K_
    monkeypatch.setattr(K_, "_pair_gemm", True)
    torch.manual_seed(M + N)
    a, b = torch.randint(-1, 2, (M, K), device="cuda").bfloat16(), torch.randint(-1, 2, (N, K), device="cuda").bfloat16()
    res, bias = torch.randint(-8, 9, (M, N), device="cuda").bfloat16(), torch.randint(-9, 10, (N + shift,), device="cuda").float()[shift:]
    z, pre = a.double() @ b.double().t() + bias.double(), torch.empty_like(res)
    close = lambda got, want, size: bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6 * size + 1e-30).all())
    cdf = lambda v: 0.5 * torch.erfc(-v / 2 ** 0.5)
    got = K_.gemm_bf16(a, b, bias=bias, residual=res, gelu=True, pre_gelu_out=pre)
    assert torch.equal(pre, z.bfloat16()) and close(got, z * cdf(z) + res.double(), z.abs())
    x = (torch.randn(M, N, device="cuda") * 2).bfloat16()
    xd = x.double()
    got = K_.gemm_bf16(a, b, bias=bias, residual=res, gelu_grad_of=x)
    assert close(got, z * (cdf(xd) + xd * torch.exp(-0.5 * xd * xd) / (2 * 3.141592653589793) ** 0.5) + res.double(), z.abs())
    own = res.clone()
    K_.gemm_bf16(a, b, residual=own, out=own, bias=bias)
    assert torch.equal(own, (z + res.double()).bfloat16())
    K_.check_errors()


@pytest.mark.parametrize("M,N,K", [(1024, 256, 64), (1100, 1120, 192), (2100, 544, 576), (9500, 1024, 64), (19000, 512, 128), (40000, 64 * 9, 64)])
def test_pair_gemm_side_operands_of_whole_numbers(M, N, K, monkeypatch):
    """The side operand is fetched a block ahead, also across tiles, and sixteen warps share eight or four blocks of columns: one tile per
    pair and several, halves in the last round, ragged edges. Residuals: whole numbers, exact. GELU': against float64, its argument
    the same bf16 numbers; the product is exact, so that what is left is bf16's rounding and the factor's approximation."""
    from gcow_b200.ops import kernels as K_
    monkeypatch.setattr(K_, "_pair_gemm", True)
    torch.manual_seed(M + N + K)
    a, b = torch.randint(-1, 2, (M, K), device="cuda").bfloat16(), torch.randint(-1, 2, (N, K), device="cuda").bfloat16()
    res = torch.randint(-8, 9, (M, N), device="cuda").bfloat16()
    prod = a.double() @ b.double().t()
    assert torch.equal(K_.gemm_bf16(a, b, residual=res), (prod + res.double()).bfloat16())
    x = (torch.randn(M, N, device="cuda") * 2).bfloat16()
    xd = x.double()
    factor = 0.5 * (1 + torch.erf(xd / 2 ** 0.5)) + xd * torch.exp(-0.5 * xd * xd) / (2 * 3.141592653589793) ** 0.5
    for r in (None, res):
        want = prod * factor + (r.double() if r is not None else 0)
        got = K_.gemm_bf16(a, b, gelu_grad_of=x, residual=r).double()
        # the approximation of Phi is good to 1.5e-7, its fp32 evaluation to a few 2^-24; |product| is at most K
        assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6 * prod.abs() + 1e-30).all())
    if N % 64 == 0:
        assert torch.equal(K_.gemm_bf16(a, b.t().contiguous(), b_t=True, residual=res), (prod + res.double()).bfloat16())
    K_.check_errors()
