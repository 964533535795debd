"""The extension module's layer functions inside autograd: saved-tensor hooks, in-place checks, lifetimes, tracing."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cases(weight_grad=True):
    from gcow_b200.ops import kernels as K
    from gcow_b200.ops import nn as gnn
    torch.manual_seed(0)

    def r(*s, dtype=torch.bfloat16):
        return torch.randn(*s, device="cuda", dtype=dtype).requires_grad_(weight_grad or dtype == torch.bfloat16)

    def nhwc(*s):
        return torch.randn(*s, device="cuda", dtype=torch.bfloat16).to(memory_format=torch.channels_last).requires_grad_(True)
    f = torch.float32
    bn = gnn.BatchNorm2d(64).cuda().requires_grad_(weight_grad)
    w, w1, w2 = r(64, 128, dtype=f), r(256, 128, dtype=f), r(128, 256, dtype=f)
    b, b1, b2 = r(64, dtype=f), r(256, dtype=f), r(128, dtype=f)
    gam, c1, c3 = r(128, dtype=f), r(64, 64, 1, 1, dtype=f), r(64, 64, 3, 3, dtype=f)
    return {
        "linear": (lambda x: K.linear(x, w, b), r(2, 64, 128)),
        "ffn": (lambda x: K.ffn_residual(x, w1, b1, w2, b2), r(2, 64, 128)),
        "layernorm": (lambda x: K.layernorm(x, gam, b2, 1e-5), r(2, 64, 128)),
        "attention": (K.fused_attention, r(2, 128, 3, 2, 64)),
        "conv1x1": (lambda x: K.conv1x1(x, c1, None), nhwc(2, 64, 8, 8)),
        "conv3x3": (lambda x: K.conv_igemm(x, c3, None, (1, 1)), nhwc(2, 64, 8, 8)),
        "batchnorm": (lambda x: K.batchnorm_act(x, bn, relu=True), nhwc(2, 64, 8, 8)),
    }


NAMES = ("linear", "ffn", "layernorm", "attention", "conv1x1", "conv3x3", "batchnorm")


@pytest.mark.parametrize("name", NAMES)
def test_saved_tensor_hooks(name):
    """Everything kept for the backward pass goes through the hooks, so offload and checkpointing see it."""
    fn, x = _cases()[name]
    packed = []

    def pack(t):
        packed.append(t.numel())
        return t.detach().cpu()
    want = torch.autograd.grad(fn(x).float().square().sum(), x)[0]
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = fn(x)
    assert packed
    got = torch.autograd.grad(y.float().square().sum(), x)[0]
    assert torch.equal(got, want)


@pytest.mark.parametrize("name", NAMES)
def test_inplace_write_is_noticed(name):
    fn, leaf = _cases()[name]
    x = leaf * 1.0
    y = fn(x)
    with torch.no_grad():
        x.mul_(2)
    with pytest.raises(RuntimeError, match="in-?place"):
        y.float().sum().backward()


@pytest.mark.parametrize("name", NAMES)
def test_graph_without_backward_is_freed(name):
    fn, x = _cases()[name]
    fn(x)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    for _ in range(3):
        fn(x)
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == before


@pytest.mark.parametrize("name", NAMES)
def test_second_backward_and_transforms_are_refused(name):
    fn, x = _cases()[name]
    y = fn(x)
    y.float().sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.backward(torch.ones_like(y))
    import torch.autograd.forward_ad as fwd
    with pytest.raises((NotImplementedError, RuntimeError)), fwd.dual_level():
        fn(fwd.make_dual(x.detach(), torch.ones_like(x)))
    with pytest.raises(RuntimeError):
        torch.func.vmap(fn)(x.detach()[None])


@pytest.mark.parametrize("name", NAMES)
def test_trace(name):
    """A traced function computes from its input, forward and backward, and not from the tracing input's result."""
    fn, x = _cases(False)[name]
    traced = torch.jit.trace(fn, (x.detach(),), check_trace=False)
    x2 = (x.detach() * 0.5 + 0.1).requires_grad_(True)
    y, z = fn(x2), traced(x2)
    assert torch.equal(y, z)
    gy = torch.randn_like(y)
    assert torch.equal(torch.autograd.grad(y, x2, gy)[0], torch.autograd.grad(z, x2, gy)[0])


def test_wrong_arguments_are_refused():
    from gcow_b200.ops import kernels as K
    x, w = torch.randn(64, 128, device="cuda").bfloat16(), torch.randn(64, 128, device="cuda")
    with pytest.raises(TypeError):
        K.linear(x, w, "b")
    with pytest.raises(RuntimeError):
        K.linear(x, w, torch.zeros(32, device="cuda"))
    with pytest.raises(RuntimeError):
        K.linear_residual(x, w, None, torch.zeros(32, 64, device="cuda"))


@pytest.mark.parametrize("rows,n,k", [(2 * 64, 64, 128), (1024, 768, 256), (1192, 320, 448)])
def test_forked_linear(rows, n, k):
    """Both gradients of the input, one of them, and a second gradient that is no contiguous matrix; hooks keep the module's own call."""
    from gcow_b200.ops import kernels as K
    from gcow_b200.ops import nn as gnn
    torch.manual_seed(rows)
    lin = gnn.Linear(k, n).cuda()
    x = torch.randn(rows, k, device="cuda").bfloat16().requires_grad_(True)
    gy, gz = torch.randn(rows, n, device="cuda").bfloat16(), torch.randn(k, rows, device="cuda").bfloat16().t()
    y, z = gnn.linear_fork(x, lin)
    assert z is not x and z.data_ptr() == x.data_ptr() and torch.equal(y, K.linear(x, lin.weight, lin.bias))
    got = torch.autograd.grad((y, z), (x, lin.weight, lin.bias), (gy, gz), retain_graph=True)
    want = torch.autograd.grad(K.linear(x, lin.weight, lin.bias), (x, lin.weight, lin.bias), gy)
    exact = gy.double() @ lin.weight.detach().bfloat16().double() + gz.double()
    # fp32 sums of k products and one bf16 rounding (2^-9 of the value; the sums' part is far below)
    assert ((got[0].double() - exact).abs() <= exact.abs() * 2.0 ** -8 + 1e-4 * exact.abs().max()).all()
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    assert torch.equal(torch.autograd.grad(y, x, gy, retain_graph=True)[0], want[0])
    assert torch.equal(torch.autograd.grad(z, x, gz)[0], gz)
    seen = []
    handle = lin.register_forward_hook(lambda m, i, o: seen.append(o.shape))
    y, z = gnn.linear_fork(x, lin)
    handle.remove()
    assert z is x and seen == [y.shape]
    y, z = gnn.linear_fork(x.detach(), lin)
    assert z.grad_fn is None and y.grad_fn is not None
    K.check_errors()


@pytest.mark.parametrize("which", ["x", "again"])
def test_forked_linear_sees_changes_in_place(which):
    """Both tensors are the memory that the weight gradient reads, so a change of either between the passes is an error, as with torch's own layers."""
    from gcow_b200.ops import kernels as K
    from gcow_b200.ops import nn as gnn
    lin = gnn.Linear(128, 64).cuda()
    x = torch.randn(128, 128, device="cuda", requires_grad=True).bfloat16()
    y, z = gnn.linear_fork(x, lin)
    assert z._version == x._version
    with torch.no_grad():
        (x if which == "x" else z).mul_(2)
    assert z._version == x._version > 0
    with pytest.raises(RuntimeError, match="modified (by an )?inplace"):
        (y.sum() + z.sum()).backward()
    y, z = gnn.linear_fork(x.detach().requires_grad_(True), lin)
    z = torch.relu_(z)                                       # with its history
    with pytest.raises(RuntimeError, match="modified (by an )?inplace"):
        (y.sum() + z.sum()).backward()
    K.check_errors()


@pytest.mark.parametrize("which", [0, 1])
def test_forked_batchnorm_sees_changes_in_place(which):
    """A consumer of one of the two results has saved the memory of both."""
    from gcow_b200.ops import kernels as K
    from gcow_b200.ops import nn as gnn
    bn = gnn.BatchNorm2d(64).cuda()
    x = torch.randn(4, 64, 9, 9, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last).requires_grad_(True)
    pair = bn(x, relu=True, fork=True)
    assert pair[0].data_ptr() == pair[1].data_ptr() and pair[0]._version == pair[1]._version
    kept = pair[1 - which] ** 2
    pair[which].add_(1)
    assert pair[0]._version == pair[1]._version > 0
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        kept.sum().backward()
    K.check_errors()


def _grads(net, x, run):
    y = run(x)
    y.backward(torch.ones_like(y))
    out = [y.detach(), x.grad] + [p.grad for p in net.parameters()]
    x.grad = None
    net.zero_grad(set_to_none=True)
    return out


@pytest.mark.parametrize("name", NAMES)
def test_checkpoint_recomputes_with_history(name):
    """Non-reentrant checkpointing reruns the region from the layer function's unpacking: operators of torch in front of
    it have to record their history there as in the first run."""
    from torch.utils.checkpoint import checkpoint
    fn, x = _cases()[name]

    def region(t):
        return fn(torch.tanh(t))
    want = torch.autograd.grad(region(x).float().square().sum(), x)[0]
    got = torch.autograd.grad(checkpoint(region, x, use_reentrant=False).float().square().sum(), x)[0]
    assert torch.equal(got, want)


@pytest.mark.parametrize("S", [128, 72])
def test_checkpoint_of_a_bert_layer(S):
    """With the fused attention and with the unfused one."""
    from torch.utils.checkpoint import checkpoint
    from gcow_b200.models.bert import BertConfig, BertLayer
    torch.manual_seed(1)
    net = BertLayer(BertConfig(hidden=128, heads=2, ffn=512)).cuda()
    x = torch.randn(2, S, 128, device="cuda").bfloat16().requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = _grads(net, x, net)
        got = _grads(net, x, lambda t: checkpoint(net, t, use_reentrant=False))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("stride", [1, 2])
def test_checkpoint_of_a_resnet_block(stride):
    from torch.utils.checkpoint import checkpoint
    from gcow_b200.models.resnet import Bottleneck
    from gcow_b200.ops import nn as gnn
    torch.manual_seed(1)
    down = torch.nn.Sequential(gnn.Conv2d(64, 256, 1, stride=stride, bias=False), gnn.BatchNorm2d(256))
    net = Bottleneck(64, 64, stride, down).cuda().to(memory_format=torch.channels_last)
    x = torch.randn(4, 64, 16, 16, device="cuda").bfloat16().to(memory_format=torch.channels_last).requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = _grads(net, x, net)
        got = _grads(net, x, lambda t: checkpoint(net, t, use_reentrant=False))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name", ["linear", "ffn", "conv1x1", "conv3x3", "batchnorm"])
def test_gradient_target(name):
    """A weight gradient goes into the tensor left in _gcow_grad_view where that fits, once per step, and nowhere near it where
    gradients accumulate, the address is not aligned or the layout differs."""
    from gcow_b200.ops import kernels as K
    fn, x = _cases()[name]
    y = fn(x)
    weights = [v for v in _leaves(y) if v is not x and v.dim() != 1 or name == "batchnorm" and v.dim() == 1]
    for w in weights:
        if w.dim() == 4:                                         # as a model in channels-last memory has them
            w.data = w.data.to(memory_format=torch.channels_last)
    fn(x).float().square().sum().backward()
    want = [w.grad.clone() for w in weights]

    def step(left):
        for w, v in zip(weights, left):
            w._gcow_grad_view = v
        hits = K.grad_view_hits()
        fn(x).float().square().sum().backward()
        return K.grad_view_hits() - hits

    def fresh():
        for w in weights:
            w.grad = None
        return [torch.full_like(w, 7.0) for w in weights]
    left = fresh()
    assert step(left) == len(weights)
    for w, v, g in zip(weights, left, want):
        assert w.grad.data_ptr() == v.data_ptr() and torch.equal(w.grad, g)
    left = [torch.full_like(w, 7.0) for w in weights]            # .grad is there: it has to be added to
    assert step(left) == 0
    for w, v, g in zip(weights, left, want):
        assert torch.equal(w.grad, 2 * g) and bool((v == 7).all())
    if name != "batchnorm":                                      # its kernel writes single floats
        fresh()
        held = [torch.full((w.numel() + 1,), 7.0, device="cuda") for w in weights]
        left = [h[1:].as_strided(w.shape, w.stride()) for h, w in zip(held, weights)]
        assert step(left) == 0
        for w, h, g in zip(weights, held, want):
            assert torch.equal(w.grad, g) and bool((h == 7).all())
    left = fresh()
    for w, v in zip(weights, left):
        w._gcow_grad_view = v
    hits = K.grad_view_hits()
    (fn(x).float().square().sum() + fn(x).float().square().sum()).backward()
    assert K.grad_view_hits() - hits <= len(weights)             # the second use of a weight has no target
    for w, g in zip(weights, want):
        assert torch.equal(w.grad, 2 * g)


def _leaves(y):
    seen, out, todo = set(), [], [y.grad_fn]
    while todo:
        f = todo.pop()
        if f is None or f in seen:
            continue
        seen.add(f)
        if hasattr(f, "variable"):
            out.append(f.variable)
        todo += [n for n, _ in f.next_functions]
    return out
