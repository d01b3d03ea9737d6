"""The work whose speed counts: training steps of the model families this framework ships, and of their single
blocks, each through the define-then-run API (``ad.*_op`` graph, ``ad.gradients`` or ``Optimizer.minimize``, an
executor, ``run(feed_dict)``) on inputs that are already on the GPU.

Steps of fixed shape are replayed from a CUDA graph (``use_graph=True``), the way the launch-bound examples are run;
the first pass of an executor runs operator by operator and the second one captures.  Everything is fp32 storage with
TF32 tensor-core products.  ``exact`` restates every network in plain torch in 64 bits.
"""
import math
import zlib

import torch
import torch.nn.functional as F

from tsplit_b200 import ndarray, optimizer
from tsplit_b200 import gpu_ops as ad
from tsplit_b200 import models
from tsplit_b200.models.resnet import bottleneck

BN_EPS, LN_EPS = 0.01, 1e-5
LR, ADAM_LR = 0.01, 1e-4


# ---------------------------------------------------------------------------------------------------- the cases
def conv(n, c, hw, kernels, widths, strides, pool, input_grad, **kw):
    return dict(kind="conv", n=n, c=c, hw=hw, kernels=kernels, widths=widths, strides=strides, pool=pool,
                input_grad=input_grad, **kw)


def transformer(n, src, tgt, d, heads, ff, vocab, blocks, **kw):
    return dict(kind="transformer", n=n, src=src, tgt=tgt, d=d, heads=heads, ff=ff, vocab=vocab, blocks=blocks, **kw)


def listed():
    return [
        # the 784-256-256-10 network on MNIST-sized input: the smallest step, all launches and latency
        dict(name="mlp_step", kind="mlp", n=64),
        # the row-by-row MNIST LSTM: some thousand dependent launches on tiny operands
        dict(name="lstm_step", kind="lstm", n=128, steps=28, features=28, hidden=128),
        # VGG's first block on RGB images: the few-channel stem and the 64-channel convolution at full resolution
        conv(16, 3, 224, "3x3,3x3", "64,64", "1,1", "max2", False, name="vgg_block1"),
        # a middle VGG layer, forward, data gradient and filter gradient: the wide 3x3 convolution
        conv(32, 256, 56, "3x3", "256", "1", "none", True, name="conv_256"),
        # a branch of Inception-B: asymmetric kernels, 17 x 17 pixels, widths that are no power of two
        conv(32, 192, 17, "1x7,7x1", "224,256", "1,1", "none", True, name="inception_1x7_7x1"),
        # ResNet's stem: 7x7 stride 2 on RGB and the overlapping 3x3 stride-2 max pool
        conv(32, 3, 224, "7x7", "64", "2", "max3", False, name="resnet_stem"),
        # the first bottleneck of ResNet-50's second stage: 1x1, 3x3 stride 2, 1x1, the strided projection, residual add
        dict(name="bottleneck_s2", kind="bottleneck", n=32, c=256, mid=128, stride=2, hw=56),
        # one encoder and one decoder block at the Transformer example's sizes (decoder length 255)
        transformer(32, 256, 256, 512, 8, 2048, 1000, 1, name="transformer_block"),
        # the same at a small, ragged size: short sequences, few heads
        transformer(3, 37, 30, 128, 4, 512, 500, 1, name="transformer_small"),
        # embedding, output projection over the 32000-word vocabulary, label smoothing, cross-entropy and Adam
        dict(name="lm_head", kind="lm_head", n=16, length=256, d=512, vocab=32000),
        # the whole of ResNet-50 with momentum, every tensor kept
        dict(name="resnet50_step", kind="resnet", n=32, hw=224, layers=50),
        # VGG-16 under the memory planner: half of what keeping everything would take
        dict(name="vgg16_tsplit", kind="vgg", n=64, hw=224, fc=512, budget_mib=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "lstm", "conv", "conv", "conv", "bottleneck", "transformer", "transformer", "lm_head"])
    if kind == "mlp":
        return dict(kind="mlp", n=_log(rng, 1, 1024))
    if kind == "lstm":
        return dict(kind="lstm", n=_log(rng, 8, 512), steps=rng.randint(4, 28), features=28, hidden=4 * rng.randint(16, 64))
    if kind == "conv":
        form = rng.choice(["stem", "square", "pointwise", "asymmetric", "strided"])
        if form == "stem":
            hw = 8 * rng.randint(12, 28)
            if rng.random() < 0.5:
                return conv(_log(rng, 2, 32), 3, hw, "7x7", "64", "2", "max3", False)
            return conv(_log(rng, 2, 16), 3, hw, "3x3,3x3", "64,64", "1,1", "max2", False)
        c = 32 * rng.randint(1, 12) if rng.random() < 0.8 else 4 * rng.randint(4, 60)
        o = 32 * rng.randint(1, 12) if rng.random() < 0.8 else 4 * rng.randint(4, 60)
        hw = rng.randint(7, 56)
        n = max(1, min(_log(rng, 1, 64), 100000 // (hw * hw)))
        if form == "square":
            return conv(n, c, hw, "3x3", str(o), "1", rng.choice(["none", "max2"]), True)
        if form == "pointwise":
            return conv(n, c, hw, "1x1,3x3", "%d,%d" % (o, c), "1,1", "none", True)
        if form == "strided":
            return conv(n, c, 2 * (hw // 2), "3x3", str(o), "2", "none", True)
        return conv(n, c, hw, "1x7,7x1", "%d,%d" % (o, c), "1,1", "none", True)
    if kind == "bottleneck":
        mid = rng.choice([64, 128, 256])
        return dict(kind="bottleneck", n=_log(rng, 2, 32), c=mid * rng.choice([2, 4]), mid=mid, stride=rng.choice([1, 2]),
                    hw=2 * rng.randint(7, 28))
    if kind == "transformer":
        heads = rng.choice([4, 8])
        d = heads * rng.choice([32, 64])
        return transformer(_log(rng, 1, 32), rng.randint(16, 256), rng.randint(16, 256), d, heads, 4 * d, rng.randint(200, 2000), 1)
    return dict(kind="lm_head", n=_log(rng, 1, 16), length=rng.randint(32, 256), d=512, vocab=4 * rng.randint(250, 8000))


# ------------------------------------------------------------------------------------------------ inputs, weights
def _gen(name, seed):
    return torch.Generator(device="cuda").manual_seed((zlib.crc32(name.encode()) + 7919 * int(seed)) % (1 << 31))


def _normal(name, shape, seed):
    return torch.randn(tuple(shape), generator=_gen(name, seed), device="cuda")


def weight(name, shape, seed):
    """A parameter as a program meets it in training: scaled like the initialisers of the models, with biases and
    normalisation parameters that have moved away from their constants."""
    z = _normal(name, shape, seed)
    if name.endswith(("_bn_scale", "_ln_scale")):
        return 1 + 0.1 * z
    if name.endswith(("_bn_bias", "_ln_bias", "_bias", "_b")):
        return 0.1 * z
    if name == "embedding_table":
        return z * shape[1] ** -0.5
    if len(shape) == 4:
        return z * math.sqrt(2.0 / (shape[1] * shape[2] * shape[3]))
    return z * math.sqrt(2.0 / (shape[0] + shape[1]))


def _labels(name, rows, classes, seed):
    return torch.randint(0, classes, (rows,), generator=_gen(name, seed), device="cuda")


def _tokens(name, n, length, vocab, seed):
    """Token ids; the tail of each sentence but the longest is padding (id 0)."""
    t = torch.randint(1, vocab, (n, length), generator=_gen(name, seed), device="cuda")
    ends = torch.randint(length // 2, length + 1, (n, 1), generator=_gen(name + "_len", seed), device="cuda")
    ends[0] = length
    return torch.where(torch.arange(length, device="cuda") < ends, t, torch.zeros_like(t)).float()


def feeds(case, seed):
    """The fed values of a case by name, as fp32 tensors on the GPU."""
    k, n = case["kind"], case["n"]
    if k == "mlp":
        return {"X": torch.rand((n, 784), generator=_gen("X", seed), device="cuda"),
                "y_": F.one_hot(_labels("y", n, 10, seed), 10).float()}
    if k == "lstm":
        return {"X": torch.rand((n, case["steps"] * case["features"]), generator=_gen("X", seed), device="cuda"),
                "y_": F.one_hot(_labels("y", n, 10, seed), 10).float()}
    if k in ("conv", "bottleneck"):
        x = _normal("X", (n, case["c"], case["hw"], case["hw"]), seed)
        return {"X": x if case["c"] == 3 else x.clamp_(min=0), "y_": F.one_hot(_labels("y", n, 16, seed), 16).float()}
    if k in ("resnet", "vgg"):
        return {"X": _normal("X", (n, 3, case["hw"], case["hw"]), seed),
                "y_": F.one_hot(_labels("y", n, 1000, seed), 1000).float()}
    if k == "transformer":
        ys = _tokens("ys", n, case["tgt"] + 1, case["vocab"], seed)
        return {"xs": _tokens("xs", n, case["src"], case["vocab"], seed), "ys_in": ys[:, :-1].contiguous(),
                "ys_out": ys[:, 1:].contiguous()}
    ys = _tokens("ys", n, case["length"] + 1, case["vocab"], seed)
    return {"ys_in": ys[:, :-1].contiguous(), "ys_out": ys[:, 1:].contiguous()}


# ---------------------------------------------------------------------------------------------------- the graphs
def _device_array(t, ctx):
    a = ndarray.empty(tuple(t.shape), ctx, use_pool=False)
    a.t.copy_(t)
    return a


class _Weights(object):
    """Parameter source of the model-building functions (``get`` / ``he``) whose values are made on the GPU."""

    def __init__(self, ctx, seed):
        self.ctx, self.seed, self.variables = ctx, seed, []

    def get(self, name, shape, scale=None, const=None):
        v = ad.Variable(name=name, value=_device_array(weight(name, shape, self.seed), self.ctx))
        self.variables.append(v)
        return v

    def he(self, name, shape, fan_in):
        return self.get(name, shape)


def _kernels(case):
    ks = [tuple(int(v) for v in k.split("x")) for k in case["kernels"].split(",")]
    return list(zip(ks, [int(v) for v in case["widths"].split(",")], [int(v) for v in case["strides"].split(",")]))


def _out(hw, k, p, s):
    return (hw + 2 * p - k) // s + 1


def _classifier(p, x, c, hw, y_):
    x = ad.array_reshape_op(ad.avg_pool2d_op(x, kernel_H=hw[0], kernel_W=hw[1], padding=0, stride=hw[0]), (-1, c))
    y = ad.matmul_op(x, p.get("fc_weight", (c, 16)))
    return y, ad.softmaxcrossentropy_op(y, y_)


def _conv_net(case, p, X, y_):
    x, c, hw = X, case["c"], (case["hw"], case["hw"])
    for i, ((kh, kw), o, s) in enumerate(_kernels(case)):
        w = p.get("conv%d_weight" % i, (o, c, kh, kw))
        x = ad.conv2d_op(x, w, padding=kh // 2, padding2=kw // 2, stride=s)
        x = ad.batch_normalization_relu_op(x, p.get("conv%d_bn_scale" % i, (1, o, 1, 1)), p.get("conv%d_bn_bias" % i, (1, o, 1, 1)))
        c, hw = o, (_out(hw[0], kh, kh // 2, s), _out(hw[1], kw, kw // 2, s))
    if case["pool"] != "none":
        k, pad = (2, 0) if case["pool"] == "max2" else (3, 1)
        x = ad.max_pool2d_op(x, kernel_H=k, kernel_W=k, padding=pad, stride=2)
        hw = tuple(_out(v, k, pad, 2) for v in hw)
    return _classifier(p, x, c, hw, y_)


def prepare(case, seed):
    ctx = ndarray.gpu(0)
    kind = case["kind"]
    fed = {k: _device_array(v, ctx) for k, v in feeds(case, seed).items()}
    state = {"fed": fed}
    if kind in ("conv", "bottleneck"):
        X, y_ = ad.Variable(name="X"), ad.Variable(name="y_")
        p = _Weights(ctx, seed)
        if kind == "conv":
            y, loss = _conv_net(case, p, X, y_)
        else:
            x, c = bottleneck(p, X, case["c"], case["mid"], case["stride"], "block")
            hw = case["hw"] // case["stride"]
            y, loss = _classifier(p, x, c, (hw, hw), y_)
        grads = ad.gradients(loss, p.variables + ([X] if case.get("input_grad", True) else []))
        nodes, extra = [loss, y] + grads, []
        feed = {X: fed["X"], y_: fed["y_"]}
    elif kind == "transformer":
        m = models.transformer(vocab_size=case["vocab"], d_model=case["d"], num_heads=case["heads"], d_ff=case["ff"],
                               num_blocks=case["blocks"], maxlen1=case["src"], maxlen2=case["tgt"] + 1, batch_size=case["n"])
        _refresh(m.variables, ctx, seed)
        # the gradient of a key projection's bias is zero but for rounding (the soft-max does not see it)
        grads = ad.gradients(m.loss, [v for v in m.variables if not v.name.endswith("_k_bias")])
        nodes, extra = [m.loss, m.logits] + grads, []
        feed = {m.xs: fed["xs"], m.ys_in: fed["ys_in"], m.ys_out: fed["ys_out"]}
    elif kind == "lm_head":
        tok, lab = ad.Variable("tokens"), ad.Variable("labels")
        p = _Weights(ctx, seed)
        table = p.get("embedding_table", (case["vocab"], case["d"]))
        scale, bias = p.get("head_ln_scale", (case["d"],)), p.get("head_ln_bias", (case["d"],))
        h = ad.layer_normalization_op(ad.embedding_lookup_op(table, tok) * case["d"] ** 0.5, scale, bias)
        logits = ad.matmul_op(ad.array_reshape_op(h, (-1, case["d"])), table, trans_B=True)
        onehot = ad.array_reshape_op(ad.one_hot_op(lab, case["vocab"]), (-1, case["vocab"]))
        smooth = ad.addbyconst_op(ad.mul_byconst_op(onehot, 0.9), 0.1 / case["vocab"])
        loss = ad.softmaxcrossentropy_op(logits, smooth)
        opt = optimizer.AdamOptimizer(ADAM_LR, ctx=ctx)
        nodes = [loss, logits, opt.minimize(loss)]
        at = [opt.tensors.index(v) for v in (scale, bias, table)]
        extra = [a[i].t for a in (opt.params,) + opt.slots() for i in at]
        feed = {tok: fed["ys_in"], lab: fed["ys_out"]}
    else:
        m = {"mlp": lambda: models.mlp(),
             "lstm": lambda: models.lstm(steps=case["steps"], features=case["features"], hidden=case["hidden"]),
             "resnet": lambda: models.resnet(case["layers"], image=case["hw"]),
             "vgg": lambda: models.vgg(16, image=case["hw"], fc_width=case["fc"])}[kind]()
        _refresh(m.variables, ctx, seed)
        opt = optimizer.MomentumOptimizer(LR, 0.9, ctx=ctx) if kind in ("resnet", "vgg") else optimizer.SGDOptimizer(LR, ctx=ctx)
        nodes = [m.loss, m.y, opt.minimize(m.loss)]
        by_name = {v.name: v.tensor_value.t for v in opt.tensors}
        extra = [by_name[k] for k in _returned(by_name)]
        feed = {m.X: fed["X"], m.y_: fed["y_"]}
    if kind == "vgg":
        state["executor"] = ad.microopExecutor(nodes, ctx=ctx, budget_bytes=case["budget_mib"] << 20, use_graph=True)
    else:
        state["executor"] = ad.Executor(nodes, ctx=ctx, use_graph=True)
    state["feed"], state["extra"] = feed, extra
    return state


def _returned(names):
    """The updated parameters that a step returns, in order: all of a small network's; of a deep one the products'
    weights at both ends (an output for each of 160 parameters would say no more)."""
    names = sorted(names)
    if len(names) <= 24:
        return names
    names = [k for k in names if k.endswith("_weight")]
    return names[:12] + names[-12:]


def _refresh(variables, ctx, seed):
    for v in variables:
        v.tensor_value = _device_array(weight(v.name, tuple(v.tensor_value.shape), seed), ctx)


def run(state):
    out = state["executor"].run(state["feed"])
    return [o.t for o in out if o is not None] + state["extra"]


# -------------------------------------------------------------------------------------------- the floor of a case
def _conv_work(case):
    """(forward flops, those of the first layer, parameters, pixels of the last map, its width)"""
    flops, first, params, c, hw = 0.0, None, 0, case["c"], (case["hw"], case["hw"])
    for (kh, kw), o, s in _kernels(case):
        hw = (_out(hw[0], kh, kh // 2, s), _out(hw[1], kw, kw // 2, s))
        f = 2.0 * case["n"] * hw[0] * hw[1] * o * c * kh * kw
        first = f if first is None else first
        flops, params, c = flops + f, params + o * c * kh * kw + 2 * o, o
    return flops, first, params, c


def work(case):
    """Flops of the products of one step; bytes: fed values and parameters read, results written, once each."""
    k, n = case["kind"], case["n"]
    if k == "mlp":
        params = 784 * 256 + 256 * 256 + 2560
        return {"flops": 2.0 * n * (3 * params - 784 * 256), "bytes": 4.0 * (n * 804 + 2 * params)}
    if k == "lstm":
        f, h = case["features"], case["hidden"]
        gates = 4 * (f * h + h * h)
        return {"flops": 2.0 * n * case["steps"] * (2 * gates + 4 * h * h), "bytes": 4.0 * (n * case["steps"] * f + 2 * (gates + 4 * h + 10 * h))}
    if k == "conv":
        flops, first, params, c = _conv_work(case)
        x = n * case["c"] * case["hw"] ** 2
        return {"flops": 3 * flops - (0 if case["input_grad"] else first), "bytes": 4.0 * (x * (2 if case["input_grad"] else 1) + 2 * (params + 16 * c))}
    if k == "bottleneck":
        c, m, s, hw = case["c"], case["mid"], case["stride"], case["hw"]
        px, py = n * hw * hw, n * (hw // s) ** 2
        proj = s != 1 or c != 4 * m
        mac = px * c * m + py * m * m * 9 + py * m * 4 * m + (py * c * 4 * m if proj else 0)
        params = c * m + 9 * m * m + 4 * m * m + (4 * m * c if proj else 0)
        return {"flops": 6.0 * mac, "bytes": 4.0 * (2 * px * c + 2 * params)}
    if k == "transformer":
        d, ff, s, t, v = case["d"], case["ff"], case["src"], case["tgt"], case["vocab"]
        rows = n * (s + 2 * t)              # self-attention of both sides and the decoder's queries over the encoder
        mac = case["blocks"] * (n * d * d * (4 * s + 4 * t + 2 * t + 2 * s) + n * d * ff * 2 * (s + t)
                                + 2 * n * d * (s * s + t * t + t * s)) + n * t * d * v
        params = case["blocks"] * (12 * d * d + 4 * d * ff) + v * d
        return {"flops": 6.0 * mac, "bytes": 4.0 * (rows + n * t * v + 2 * params)}
    if k == "lm_head":
        r, p = n * case["length"], case["d"] * case["vocab"]
        return {"flops": 6.0 * r * p, "bytes": 4.0 * (2 * r + r * case["vocab"] + 6 * p)}
    mac, params = _resnet_work(case) if k == "resnet" else _vgg_work(case)
    return {"flops": 6.0 * n * mac, "bytes": 4.0 * (3 * n * case["hw"] ** 2 + 4 * params)}


def _resnet_layers(case):
    """(name, in, out, kernel, stride, relu, map size of its input) of every convolution."""
    hw = _out(case["hw"], 7, 3, 2)
    yield "resnet_stem", 3, 64, 7, 2, case["hw"]
    hw, cin = _out(hw, 3, 1, 2), 64
    for s, reps in enumerate({50: [3, 4, 6, 3], 26: [2, 2, 2, 2]}[case["layers"]]):
        for r in range(reps):
            mid, st = 64 << s, 2 if (r == 0 and s > 0) else 1
            name = "resnet_s%d_b%d" % (s + 1, r + 1)
            yield name + "_a", cin, mid, 1, 1, hw
            yield name + "_b", mid, mid, 3, st, hw
            yield name + "_c", mid, 4 * mid, 1, 1, hw // st
            if st != 1 or cin != 4 * mid:
                yield name + "_proj", cin, 4 * mid, 1, st, hw
            cin, hw = 4 * mid, hw // st


def _resnet_work(case):
    mac, params = 2048 * 1000, 2048 * 1000
    for _, c, o, k, s, hw in _resnet_layers(case):
        mac += o * c * k * k * (hw // s) ** 2
        params += o * c * k * k + 2 * o
    return mac, params


def _vgg_work(case):
    mac, params, c, hw = 0, 0, 3, case["hw"]
    for reps, o in zip([2, 2, 3, 3, 3], [64, 128, 256, 512, 512]):
        for _ in range(reps):
            mac += o * c * 9 * hw * hw
            params += o * c * 9 + 2 * o
            c = o
        hw //= 2
    fc = hw * hw * c * case["fc"] + case["fc"] ** 2 + case["fc"] * 1000
    return mac + fc, params + fc


def tolerance(case):
    """TF32 operands carry 10 mantissa bits, the same ones in any correct implementation; what may differ is the order
    of the 32-bit sums, and through them ReLU masks of values at zero and the maxima of pooling windows."""
    return {"mlp": {"rel": 2e-4, "max": 0.05}, "lstm": {"rel": 2e-4, "max": 0.05}, "conv": {"rel": 4e-3, "max": 0.5},
            "bottleneck": {"rel": 4e-3, "max": 0.5}, "transformer": {"rel": 2e-3, "max": 0.2},
            "lm_head": {"rel": 2e-3, "max": 0.2}, "resnet": {"rel": 1e-2, "max": 0.5}, "vgg": {"rel": 1e-2, "max": 0.5}}[case["kind"]]


# --------------------------------------------------------------------------------------- the same in 64-bit torch
class _Exact(object):
    def __init__(self, seed):
        self.seed, self.leaves = seed, {}

    def __call__(self, name, shape):
        if name not in self.leaves:
            self.leaves[name] = weight(name, shape, self.seed).double().requires_grad_()
        return self.leaves[name]


def _bn(w, x, name, relu):
    o = x.shape[1]
    y = F.batch_norm(x, None, None, w(name + "_bn_scale", (1, o, 1, 1)).reshape(-1), w(name + "_bn_bias", (1, o, 1, 1)).reshape(-1), True, 0.0, BN_EPS)
    return F.relu(y) if relu else y


def _conv_bn(w, x, o, kh, kw, stride, name, relu=True):
    y = F.conv2d(x, w(name + "_weight", (o, x.shape[1], kh, kw)), stride=stride, padding=(kh // 2, kw // 2))
    return _bn(w, y, name, relu)


def _bottleneck(w, x, mid, stride, name):
    y = _conv_bn(w, x, mid, 1, 1, 1, name + "_a")
    y = _conv_bn(w, y, mid, 3, 3, stride, name + "_b")
    y = _conv_bn(w, y, 4 * mid, 1, 1, 1, name + "_c", relu=False)
    if stride != 1 or x.shape[1] != 4 * mid:
        x = _conv_bn(w, x, 4 * mid, 1, 1, stride, name + "_proj", relu=False)
    return F.relu(x + y)


def _cross_entropy(y, target):
    return -(target * F.log_softmax(y, 1)).sum(1).mean().reshape(1)


def _positions(length, d):
    i = torch.arange(d, device="cuda")
    a = torch.arange(length, device="cuda").double()[:, None] / torch.pow(10000.0, ((i // 2) * 2).double() / d)
    return torch.where(i % 2 == 0, torch.sin(a), torch.cos(a)).float().double()


def _transformer_exact(case, w, f):
    d, h, ff, n = case["d"], case["heads"], case["ff"], case["n"]
    table = w("embedding_table", (case["vocab"], d))

    def dense(x, a, b, name):
        return x @ w(name + "_weight", (a, b)) + w(name + "_bias", (b,))

    def norm(x, name):
        return F.layer_norm(x, (d,), w(name + "_ln_scale", (d,)), w(name + "_ln_bias", (d,)), LN_EPS)

    def attention(q_in, kv, name, key, causal):
        q, k, v = (dense(t, d, d, name + "_" + s).reshape(n, -1, h, d // h).transpose(1, 2) for t, s in ((q_in, "q"), (kv, "k"), (kv, "v")))
        x = q @ k.transpose(2, 3) / math.sqrt(d // h) + torch.where(key == 0, -1e9, 0.0)[:, None, None, :]
        if causal:
            x = torch.where(torch.ones(x.shape[-2:], device="cuda").tril() > 0, x, torch.full((), -1e9, dtype=x.dtype, device="cuda"))
        c = (torch.softmax(x, -1) @ v).transpose(1, 2).reshape(n, -1, d)
        return norm(dense(c, d, d, name + "_o") + q_in, name)

    def feed_forward(x, name):
        return norm(dense(F.relu(dense(x, d, ff, name + "_ff1")), ff, d, name + "_ff2") + x, name + "_ff")

    def embed(tok):
        return table[tok.long()] * d ** 0.5 + _positions(tok.shape[1], d)

    enc = embed(f["xs"])
    for i in range(case["blocks"]):
        enc = feed_forward(attention(enc, enc, "enc%d_self" % i, f["xs"], False), "enc%d" % i)
    dec = embed(f["ys_in"])
    for i in range(case["blocks"]):
        dec = attention(dec, dec, "dec%d_self" % i, f["ys_in"], True)
        dec = attention(dec, enc, "dec%d_cross" % i, f["xs"], False)
        dec = feed_forward(dec, "dec%d" % i)
    return dec.reshape(-1, d) @ table.T


def _smooth(labels, vocab):
    return F.one_hot(labels.reshape(-1).long(), vocab).double() * 0.9 + 0.1 / vocab


def _adam(params, grads):
    """First step from zero moments: parameters, first and second moments."""
    b1, b2, eps = 0.9, 0.999, 1e-7
    m, v = [(1 - b1) * g for g in grads], [(1 - b2) * g * g for g in grads]
    p = [(p - ADAM_LR * (a / (1 - b1)) / (torch.sqrt(b / (1 - b2)) + eps)).detach() for p, a, b in zip(params, m, v)]
    return p + m + v


def exact(case, seed):
    kind = case["kind"]
    if kind == "vgg":
        return None                     # minutes of 64-bit convolutions
    f = {k: v.double() for k, v in feeds(case, seed).items()}
    w = _Exact(seed)
    if kind in ("conv", "bottleneck"):
        x = f["X"].requires_grad_()
        if kind == "conv":
            y = x
            for i, ((kh, kw), o, s) in enumerate(_kernels(case)):
                y = _conv_bn(w, y, o, kh, kw, s, "conv%d" % i)
            if case["pool"] != "none":
                k, pad = (2, 0) if case["pool"] == "max2" else (3, 1)
                y = F.max_pool2d(y, k, 2, pad)
        else:
            y = _bottleneck(w, x, case["mid"], case["stride"], "block")
        y = y.mean((2, 3)) @ w("fc_weight", (y.shape[1], 16))
        loss = _cross_entropy(y, f["y_"])
        leaves = list(w.leaves.values()) + ([x] if case.get("input_grad", True) else [])
        return [loss.detach(), y.detach()] + list(torch.autograd.grad(loss.sum(), leaves))
    if kind == "transformer":
        logits = _transformer_exact(case, w, f)
        loss = _cross_entropy(logits, _smooth(f["ys_out"], case["vocab"]))
        leaves = [v for k, v in w.leaves.items() if not k.endswith("_k_bias")]
        return [loss.detach(), logits.detach()] + list(torch.autograd.grad(loss.sum(), leaves))
    if kind == "lm_head":
        table, d = w("embedding_table", (case["vocab"], case["d"])), case["d"]
        scale, bias = w("head_ln_scale", (d,)), w("head_ln_bias", (d,))
        h = F.layer_norm(table[f["ys_in"].long()] * d ** 0.5, (d,), scale, bias, LN_EPS)
        logits = h.reshape(-1, d) @ table.T
        loss = _cross_entropy(logits, _smooth(f["ys_out"], case["vocab"]))
        leaves = [scale, bias, table]
        return [loss.detach(), logits.detach()] + _adam(leaves, torch.autograd.grad(loss.sum(), leaves))
    if kind == "mlp":
        x, sizes = f["X"], (784, 256, 256, 10)
        for i in range(3):
            x = x @ w("mlp_fc%d_weight" % (i + 1), (sizes[i], sizes[i + 1]))
            x = F.relu(x) if i < 2 else x
        y = x
    elif kind == "lstm":
        h = c = None
        fe, hi = case["features"], case["hidden"]
        for t in range(case["steps"]):
            xt = f["X"][:, t * fe:(t + 1) * fe]
            g = {}
            for name in ("forget", "input", "output", "cell"):
                z = xt @ w("lstm_%s_w" % name, (fe, hi)) + w("lstm_%s_b" % name, (hi,))
                u = w("lstm_%s_u" % name, (hi, hi))
                z = z if h is None else z + h @ u
                g[name] = torch.tanh(z) if name == "cell" else torch.sigmoid(z)
            c = g["input"] * g["cell"] if c is None else g["forget"] * c + g["input"] * g["cell"]
            h = g["output"] * torch.tanh(c)
        y = h @ w("lstm_dense_w", (hi, 10)) + w("lstm_dense_b", (10,))
    else:
        x = F.max_pool2d(_conv_bn(w, f["X"], 64, 7, 7, 2, "resnet_stem"), 3, 2, 1)
        for s, reps in enumerate({50: [3, 4, 6, 3], 26: [2, 2, 2, 2]}[case["layers"]]):
            for r in range(reps):
                x = _bottleneck(w, x, 64 << s, 2 if (r == 0 and s > 0) else 1, "resnet_s%d_b%d" % (s + 1, r + 1))
        y = x.mean((2, 3)) @ w("resnet_fc_weight", (x.shape[1], 1000))
    loss = _cross_entropy(y, f["y_"])
    names = _returned(w.leaves)
    grads = torch.autograd.grad(loss.sum(), [w.leaves[k] for k in names])
    return [loss.detach(), y.detach()] + [(w.leaves[k] - LR * g).detach() for k, g in zip(names, grads)]
