"""Performance cases: what users of gcow_b200 run on one B200, as calls of its public API.

Five families, each with the range of sizes and options that its users meet:

* ``codec1d``   - flat float32 vectors (gradients) through ``compress`` / ``decompress``, 1-D blocks of 4: one bias
                  vector up to a 256 MB buffer; fixed rate 2, 4, 8, 16 or 32 bits/value, fixed accuracy, fixed precision.
* ``codec2d``   - two-dimensional fields through the same two calls, 4 x 4 blocks: the reference codec's own use.
* ``allreduce`` - ``CompressedAllReduce`` of a gradient bucket. One process and one GPU, so the call is the lossy round
                  trip of the local gradient, which is what a single-GPU training run applies to every bucket.
* ``conv_bn``   - forward and backward of one Conv2d + BatchNorm2d pair, the ResNet layer shapes.
* ``bert_layer`` - forward and backward of one transformer layer at the BERT sizes.

Codec and all-reduce outputs are bit-exact by definition of the stream; layers compute in bf16.
"""
import math

import torch

import gcow_b200 as g

# Every convolution of a ResNet-50 stage: input channels, output channels, filter, stride, input height and width.
RESNET_LAYERS = (
    (64, 64, 1, 1, 56), (64, 64, 3, 1, 56), (64, 256, 1, 1, 56), (256, 64, 1, 1, 56), (256, 128, 1, 1, 56),
    (128, 128, 3, 2, 56), (128, 512, 1, 1, 28), (256, 512, 1, 2, 56), (512, 128, 1, 1, 28), (128, 128, 3, 1, 28),
    (512, 256, 1, 1, 28), (256, 256, 3, 2, 28), (256, 1024, 1, 1, 14), (512, 1024, 1, 2, 28), (1024, 256, 1, 1, 14),
    (256, 256, 3, 1, 14), (1024, 512, 1, 1, 14), (512, 512, 3, 2, 14), (512, 2048, 1, 1, 7), (1024, 2048, 1, 2, 14),
    (2048, 512, 1, 1, 7), (512, 512, 3, 1, 7),
)
# hidden size, heads, feed-forward width of bert_tiny, bert_base and bert_large
BERT_SIZES = ((128, 2, 512), (768, 12, 3072), (1024, 16, 4096))


def listed():
    return [
        # the bias gradient of a 1000-class layer: the smallest tensor anybody compresses, all latency
        dict(name="bias_roundtrip", family="codec1d", op="roundtrip", n=1000, mode="rate", level=8),
        # the 2^20-value vector of the fixed-rate configuration
        dict(name="vector_1m_roundtrip", family="codec1d", op="roundtrip", n=1 << 20, mode="rate", level=8),
        # a 256 MB gradient buffer, each direction by itself (sender and receiver)
        dict(name="buffer_256mb_encode", family="codec1d", op="encode", n=1 << 26, mode="rate", level=8),
        dict(name="buffer_256mb_decode", family="codec1d", op="decode", n=1 << 26, mode="rate", level=8),
        # a 25 MB bucket whose length is no multiple of a block, at the rate of the ImageNet study
        dict(name="bucket_ragged_roundtrip", family="codec1d", op="roundtrip", n=6_553_603, mode="rate", level=16),
        # the whole flattened ResNet-50 gradient at the ImageNet study's tolerance: the codec round trip that the
        # fixed-accuracy training mode applies
        dict(name="gradient_accuracy_roundtrip", family="codec1d", op="roundtrip", n=25_557_032, mode="tolerance", level=1e-6),
        # the reference codec's own call (fixed accuracy 1e-3 on a square field): its default host size and its largest
        dict(name="field_510_roundtrip", family="codec2d", op="roundtrip", ny=510, nx=510, mode="tolerance", level=1e-3),
        dict(name="field_7654_roundtrip", family="codec2d", op="roundtrip", ny=7654, nx=7654, mode="tolerance", level=1e-3),
        # a field with partial blocks on both edges at fixed rate
        dict(name="field_ragged_rate_roundtrip", family="codec2d", op="roundtrip", ny=2047, nx=3001, mode="rate", level=8),
        # one 25 MB DDP bucket
        dict(name="bucket_allreduce", family="allreduce", n=6_553_600, rate=8),
        # a 3x3 layer of the second ResNet-50 stage at the training batch of 256
        dict(name="conv_bn_3x3", family="conv_bn", batch=256, layer=9),
        # one layer of BERT-large at the training batch of 32 x 512 tokens
        dict(name="bert_large_layer", family="bert_layer", batch=32, seq=512, size=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choices(("codec1d", "codec2d", "allreduce", "conv_bn", "bert_layer"), (35, 25, 12, 14, 14))[0]
    if family == "codec1d":
        mode = rng.choices(("rate", "tolerance", "precision"), (7, 2, 1))[0]
        if mode == "rate":
            level = rng.choices((2, 4, 8, 16, 32), (1, 3, 4, 3, 1))[0]
            return dict(family=family, op=rng.choice(("encode", "decode", "roundtrip")),
                        n=_log(rng, 256, 1 << 26 if level <= 8 else 1 << 25), mode=mode, level=level)
        level = rng.choice((1e-3, 1e-6)) if mode == "tolerance" else rng.choice((8, 16))
        return dict(family=family, op=rng.choice(("decode", "roundtrip")), n=_log(rng, 256, 25_557_032), mode=mode, level=level)
    if family == "codec2d":
        mode = rng.choices(("tolerance", "rate", "precision"), (5, 4, 1))[0]
        level = {"tolerance": rng.choice((1e-1, 1e-3)), "rate": rng.choice((4, 8, 16)), "precision": rng.choice((8, 16))}[mode]
        top = 7654 if mode == "tolerance" else 4096
        op = rng.choice(("encode", "decode", "roundtrip") if mode == "rate" else ("decode", "roundtrip"))
        return dict(family=family, op=op, ny=_log(rng, 64, top), nx=_log(rng, 64, top), mode=mode, level=level)
    if family == "allreduce":
        return dict(family=family, n=_log(rng, 256, 1 << 25), rate=rng.choice((4, 8, 16)))
    if family == "conv_bn":
        return dict(family=family, batch=_log(rng, 16, 256), layer=rng.randrange(len(RESNET_LAYERS)))
    seq = rng.choice((128, 256, 384, 512, 8 * rng.randint(9, 63)))
    return dict(family=family, batch=max(1, _log(rng, 512, 16384) // seq), seq=seq, size=rng.randrange(len(BERT_SIZES)))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _gradient(n, gen):
    """Gradient values: N(0, 1e-3)."""
    return torch.randn(n, device="cuda", generator=gen) * 1e-3


def _field(ny, nx, gen):
    """The reference's test surface exp(-(x^2 + y^2)) on [0, 2)^2, centre and width moved by the seed, with measurement
    noise of 1e-4."""
    r = torch.rand(4, device="cuda", generator=gen)
    y = torch.arange(ny, device="cuda", dtype=torch.float32) * (2.0 / ny) - 0.3 * r[0]
    x = torch.arange(nx, device="cuda", dtype=torch.float32) * (2.0 / nx) - 0.3 * r[1]
    f = torch.exp(-((0.7 + 0.6 * r[2]) * x[None, :] ** 2 + (0.7 + 0.6 * r[3]) * y[:, None] ** 2))
    return f + torch.randn((ny, nx), device="cuda", generator=gen) * 1e-4


def prepare(case, seed):
    gen = _generator(seed)
    family = case["family"]
    if family in ("codec1d", "codec2d"):
        dim = 1 if family == "codec1d" else 2
        x = _gradient(case["n"], gen) if dim == 1 else _field(case["ny"], case["nx"], gen)
        how = {case["mode"]: case["level"], "dim": dim}
        state = dict(family="codec", op=case["op"], x=x, how=how, fixed=case["mode"] == "rate")
        if case["op"] == "decode":
            state["c"] = g.compress(x, **how)
        return state
    if family == "allreduce":
        from gcow_b200.comm import CompressedAllReduce
        x = _gradient(case["n"], gen)
        return dict(family=family, ar=CompressedAllReduce(case["n"], g.GcowConfig(rate=case["rate"])), x=x,
                    out=torch.empty_like(x))
    torch.manual_seed(seed)
    return _prepare_conv_bn(case, gen) if family == "conv_bn" else _prepare_bert_layer(case, gen)


def _prepare_conv_bn(case, gen):
    from gcow_b200.ops import nn as gnn
    cin, cout, k, stride, hw = RESNET_LAYERS[case["layer"]]
    conv = gnn.Conv2d(cin, cout, k, stride=stride, padding=k // 2, bias=False)
    net = torch.nn.Sequential(conv, gnn.BatchNorm2d(cout)).cuda().to(memory_format=torch.channels_last)
    with torch.no_grad():
        net[1].weight.add_(torch.randn(cout, device="cuda", generator=gen) * 0.1)
        net[1].bias.add_(torch.randn(cout, device="cuda", generator=gen) * 0.1)
    out = (hw - 1) // stride + 1

    def activation(c, s):
        t = torch.randn((case["batch"], s, s, c), device="cuda", generator=gen).to(torch.bfloat16)
        return t.permute(0, 3, 1, 2)                    # logical NCHW in channels-last memory
    return dict(family="conv_bn", net=net, x=activation(cin, hw).requires_grad_(True), gy=activation(cout, out))


def _prepare_bert_layer(case, gen):
    from gcow_b200.models.bert import BertConfig, BertLayer
    from gcow_b200.ops.optim import FusedAdamW
    hidden, heads, ffn = BERT_SIZES[case["size"]]
    net = BertLayer(BertConfig(hidden=hidden, heads=heads, ffn=ffn)).cuda()
    with torch.no_grad():
        for name, p in net.named_parameters():
            base = 1.0 if name.startswith("ln") and p is getattr(net, name.split(".")[0]).weight else 0.0
            p.copy_(base + torch.randn(p.shape, device="cuda", generator=gen) * 0.02)

    def activation():
        return torch.randn((case["batch"], case["seq"], hidden), device="cuda", generator=gen).to(torch.bfloat16)
    state = dict(family="bert_layer", net=net, x=activation().requires_grad_(True), gy=activation())
    # one optimiser step, as in the middle of a training run: the optimiser keeps bf16 copies of the weights
    run(state)
    FusedAdamW(net.parameters(), lr=1e-4).step()
    return state


def run(state):
    family = state["family"]
    if family == "codec":
        if state["op"] == "decode":
            return g.decompress(state["c"])
        c = g.compress(state["x"], **state["how"])
        if state["op"] == "encode":
            return c.stream
        y = g.decompress(c)
        # a variable-rate stream has another length for every input: the blocks' bit offsets and the values decoded from
        # all of its bits stand for it
        return [c.stream, y] if state["fixed"] else [c.index, y]
    if family == "allreduce":
        return state["ar"](state["x"], out=state["out"])
    net, x = state["net"], state["x"]
    net.zero_grad(set_to_none=True)
    x.grad = None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = net(x)
    y.backward(state["gy"])
    out = [y.detach(), x.grad] + [p.grad for p in net.parameters()]
    if family == "conv_bn":
        out += [net[1].running_mean, net[1].running_var]
    return out


def _stream_bytes(case):
    """Size of the compressed stream (with the per-block index of the variable-rate modes): exact at fixed rate, about
    right for the values that prepare() makes otherwise."""
    d2 = case["family"] == "codec2d"
    n = case["ny"] * case["nx"] if d2 else case["n"]
    if case["mode"] == "rate":
        return max(case["level"], 2.25 if not d2 else 0) * n / 8
    bits = {("tolerance", 1e-1): 1.2, ("tolerance", 1e-3): 2.5, ("precision", 8): 4.0, ("precision", 16): 10.0}[case["mode"], case["level"]] \
        if d2 else {("tolerance", 1e-3): 3.5, ("tolerance", 1e-6): 13.0, ("precision", 8): 8.0, ("precision", 16): 16.0}[case["mode"], case["level"]]
    return bits * n / 8 + 8 * (n / (16 if d2 else 4))


def work(case):
    family = case["family"]
    if family in ("codec1d", "codec2d"):
        n = case["ny"] * case["nx"] if family == "codec2d" else case["n"]
        one_way = 4 * n + _stream_bytes(case)
        return {"bytes": one_way * (2 if case["op"] == "roundtrip" else 1), "flops": 0}
    if family == "allreduce":
        return {"bytes": 8 * case["n"], "flops": 0}
    if family == "conv_bn":
        cin, cout, k, stride, hw = RESNET_LAYERS[case["layer"]]
        pin, pout = case["batch"] * hw * hw, case["batch"] * ((hw - 1) // stride + 1) ** 2
        weights = cin * cout * k * k
        # x, y, gy, dx in bf16 and the weights and their gradient; three products
        return {"bytes": 4 * (pin * cin + pout * cout) + 6 * weights, "flops": 6 * pout * weights}
    hidden, heads, ffn = BERT_SIZES[case["size"]]
    tokens = case["batch"] * case["seq"]
    weights = 4 * hidden * hidden + 2 * hidden * ffn
    return {"bytes": 8 * tokens * hidden + 6 * weights, "flops": 6 * tokens * weights + 12 * tokens * case["seq"] * hidden}


def tolerance(case):
    if case["family"] in ("codec1d", "codec2d", "allreduce"):
        return "exact"
    return {"rel": 1e-2}
