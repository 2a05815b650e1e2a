"""Performance cases of the AM-Simulator path: what a user has the library compute.

Every case runs through the public entry points: the layers and networks
(``approxtrain_b200.layers``, ``.nets``, ``.dp``) or the ops behind them
(``approxtrain_b200.ops``).  The tables are the shipped ones; MBM_7 and MIT_7 are
what the benchmark networks train with.  Sizes are those of the networks in
``approxtrain_b200/nets.py`` and of ``bench.py``, plus ragged ones.

Kinds of cases
--------------
``mlp_infer``   LeNet-300-100 forward without gradients: three tiny fused dense
                layers, the smallest thing anyone runs (latency of the calls).
``lenet5_step`` one eager SGD step of LeNet-5 through ``DataParallelSGD``: the
                launch-bound training loop.
``conv_infer``  one inference convolution with the folded batch normalisation and
                ReLU in its epilogue.
``conv_train``  one AMConv2D layer, forward and backward (input, filter and bias
                gradient).  Its input is a ReLU output (half of it zeros) as in
                the networks, except a first layer's, which is an image and needs
                no gradient.
``dense_train`` one denseam layer, forward and backward.
``attention``   scores and context products of multi-head attention (MatMulAM),
                forward and backward.
"""
import math
import os

import torch

import approxtrain_b200
from approxtrain_b200 import layers, nets, ops
from approxtrain_b200.dp import DataParallelSGD

_LUTS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(approxtrain_b200.__file__))), "tests", "golden", "lut")
_MOST_MACS = 3 * 64 * 14 * 14 * 256 * 256 * 9        # products of the largest listed case
_MOST_MACS_DET = 3 * 16 * 28 * 28 * 128 * 128 * 9    # deterministic mode is slower per product


def _conv(name, kind, lut, n, h, w, c, kh, kw, k, stride, padding, det=False, image=False):
    return dict(name=name, kind=kind, lut=lut, n=n, h=h, w=w, c=c, kh=kh, kw=kw, k=k, stride=stride, padding=padding,
                det=det, image=image)


def listed():
    return [
        # LeNet-300-100 answering a small batch: nothing but call latency
        dict(name="mlp_infer_b16", kind="mlp_infer", lut="MBM_7", n=16, det=False),
        # the LeNet-5 training loop at its benchmark batch, step by step
        dict(name="lenet5_step_b128", kind="lenet5_step", lut="MIT_7", n=128, det=False),
        # a ResNet-50 stage-3 convolution serving one image
        _conv("conv3x3_infer_b1", "conv_infer", "MBM_7", 1, 28, 28, 128, 3, 3, 128, 1, "SAME"),
        # the ResNet-50 first layer on a training batch (three channels, no input gradient)
        _conv("stem7x7_train_b32", "conv_train", "MBM_7", 32, 230, 230, 3, 7, 7, 64, 2, "VALID", image=True),
        # ResNet-50 stage 2: many pixels, few channels
        _conv("conv3x3_56_train_b32", "conv_train", "MBM_7", 32, 55, 55, 64, 3, 3, 64, 1, "SAME"),
        # the microbenchmark's shape B: the largest
        _conv("conv3x3_14_train_b64", "conv_train", "MBM_7", 64, 14, 14, 256, 3, 3, 256, 1, "SAME"),
        # a bottleneck's expanding 1x1 layer
        _conv("conv1x1_14_train_b32", "conv_train", "MBM_7", 32, 14, 14, 256, 1, 1, 1024, 1, "VALID"),
        # a bottleneck's strided projection
        _conv("project_s2_train_b32", "conv_train", "MBM_7", 32, 55, 55, 256, 1, 1, 512, 2, "VALID"),
        # ragged everything, a narrower table
        _conv("ragged5x5_train", "conv_train", "MIT_5", 7, 27, 31, 37, 5, 5, 45, 1, "SAME"),
        # the reference's order bit by bit
        _conv("conv3x3_det_train_b8", "conv_train", "MBM_7", 8, 28, 28, 128, 3, 3, 128, 1, "SAME", det=True),
        # the Transformer's feed-forward layer over 64 x 128 tokens
        dict(name="ffn_train_8192", kind="dense_train", lut="MIT_7", rows=8192, width=512, units=2048, det=False),
        # the Transformer's attention products, 64 sequences x 8 heads
        dict(name="attention_train_b64", kind="attention", lut="MIT_7", n=64, heads=8, seq=128, depth=64, det=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    """Mostly what networks use (multiples of 16), sometimes odd counts."""
    v = _log(rng, lo, hi)
    return v if v < 16 or rng.random() < 0.3 else max(16, v // 16 * 16)


def draw(rng):
    while True:
        kind = rng.choice(["mlp_infer", "lenet5_step", "conv_infer", "conv_train", "conv_train", "conv_train", "conv_train",
                           "dense_train", "dense_train", "attention"])
        lut = rng.choice(["MBM_7", "MBM_7", "MBM_7", "MIT_7", "MIT_7", "MBM_5", "MIT_5"])
        if kind in ("mlp_infer", "lenet5_step"):
            case = dict(kind=kind, lut=lut, n=_log(rng, 1, 300), det=False)
        elif kind in ("conv_infer", "conv_train"):
            kh = kw = rng.choice([1, 1, 3, 3, 3, 5, 7])
            image = kind == "conv_train" and kh >= 5 and rng.random() < 0.5
            case = dict(kind=kind, lut=lut, n=_log(rng, 1, 8 if kind == "conv_infer" else 64), h=_log(rng, 7, 232),
                        w=_log(rng, 7, 232), c=rng.choice([1, 3]) if image else _channels(rng, 6, 1024), kh=kh, kw=kw,
                        k=_channels(rng, 6, 1024), stride=rng.choice([1, 1, 1, 2]), padding=rng.choice(["SAME", "VALID"]),
                        det=kind == "conv_train" and rng.random() < 0.15, image=image)
        elif kind == "dense_train":
            case = dict(kind=kind, lut=lut, rows=_log(rng, 16, 8192), width=_channels(rng, 64, 4096),
                        units=_channels(rng, 10, 4096), det=False)
        else:
            case = dict(kind=kind, lut=lut, n=_log(rng, 1, 64), heads=rng.choice([1, 4, 8]), seq=_log(rng, 16, 256),
                        depth=rng.choice([32, 64, 64, 128]), det=False)
        macs = _macs(case)
        if 1e5 <= macs <= (_MOST_MACS_DET if case["det"] else _MOST_MACS) and _bytes(case) < 1.2e9:
            return case


def _conv_out(case):
    if case["padding"] == "SAME":
        return -(-case["h"] // case["stride"]), -(-case["w"] // case["stride"])
    return (case["h"] - case["kh"]) // case["stride"] + 1, (case["w"] - case["kw"]) // case["stride"] + 1


def _macs(case):
    """Products of one pass (every one of them approximate)."""
    kind = case["kind"]
    if kind == "mlp_infer":
        return case["n"] * (784 * 300 + 300 * 100 + 100 * 10)
    if kind == "lenet5_step":
        first = 28 * 28 * 6 * 25                       # its input needs no gradient
        rest = 10 * 10 * 16 * 25 * 6 + 400 * 120 + 120 * 84 + 84 * 10
        return case["n"] * (2 * first + 3 * rest)
    if kind in ("conv_infer", "conv_train"):
        oh, ow = _conv_out(case)
        one = case["n"] * oh * ow * case["k"] * case["kh"] * case["kw"] * case["c"]
        return one * (1 if kind == "conv_infer" else 2 if case["image"] else 3)
    if kind == "dense_train":
        return 3 * case["rows"] * case["width"] * case["units"]
    return 6 * case["n"] * case["heads"] * case["seq"] ** 2 * case["depth"]   # two products, each with two gradients


def _bytes(case):
    """Each input read once and each output written once, FP32."""
    kind = case["kind"]
    if kind == "mlp_infer":
        return 4 * (784 * 300 + 300 + 300 * 100 + 100 + 100 * 10 + 10 + case["n"] * (784 + 10))
    if kind == "lenet5_step":
        params = 6 * 26 + 16 * 151 + 401 * 120 + 121 * 84 + 85 * 10
        return 4 * (2 * params + case["n"] * 784) + 8 * case["n"]
    if kind in ("conv_infer", "conv_train"):
        oh, ow = _conv_out(case)
        x, y = case["n"] * case["h"] * case["w"] * case["c"], case["n"] * oh * ow * case["k"]
        f = case["kh"] * case["kw"] * case["c"] * case["k"]
        if kind == "conv_infer":
            return 4 * (x + f + 2 * case["k"] + y)
        return 4 * (x * (1 if case["image"] else 2) + 2 * f + 2 * case["k"] + 2 * y)
    if kind == "dense_train":
        r, i, u = case["rows"], case["width"], case["units"]
        return 4 * (2 * r * i + 2 * i * u + 2 * u + 2 * r * u)
    b, s, d = case["n"] * case["heads"], case["seq"], case["depth"]
    return 4 * b * (8 * s * d + 4 * s * s)   # q k v o and their gradients; scores and weights each once, with gradients


def work(case):
    return {"bytes": _bytes(case), "flops": 2 * _macs(case)}


def tolerance(case):
    if case["det"]:
        return "exact"            # bit-identical to the reference's kernels: one ascending chain per output
    if case["kind"] == "lenet5_step":
        return {"rel": 1e-4}      # a ReLU or pooling decision on the edge may fall the other way
    return {"rel": 1e-5}          # FP32 sums in another order


def _lut(case):
    return os.path.join(_LUTS, case["lut"] + ".bin")


def _fill(params, gen, fan_ins):
    """He-normal weights and small biases from the case's own generator."""
    with torch.no_grad():
        for p, fan in zip(params, fan_ins):
            p.copy_(torch.randn(p.shape, generator=gen, device="cuda") * (math.sqrt(2.0 / fan) if fan else 0.01))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    kind, lut, det = case["kind"], _lut(case), case["det"]
    if kind == "mlp_infer":
        net = nets.LeNet300100(lut, deterministic=det).cuda()
        _fill(net.parameters(), gen, [784, 0, 300, 0, 100, 0])
        return dict(case=case, net=net, x=torch.rand(case["n"], 784, generator=gen, device="cuda"))
    if kind == "lenet5_step":
        net = nets.LeNet5(lut, deterministic=det).cuda()
        _fill(net.parameters(), gen, [25, 0, 150, 0, 400, 0, 120, 0, 84, 0])
        x = torch.rand(case["n"], 28, 28, 1, generator=gen, device="cuda")
        y = torch.randint(0, 10, (case["n"],), generator=gen, device="cuda")
        trainer = DataParallelSGD(net, lr=1e-3)
        return dict(case=case, net=net, trainer=trainer, loss=lambda: torch.nn.functional.cross_entropy(net(x), y))
    if kind in ("conv_infer", "conv_train"):
        n, h, w, c, kh, kw, k = (case[i] for i in ("n", "h", "w", "c", "kh", "kw", "k"))
        x = rnd(n, h, w, c) if case["image"] else torch.relu(rnd(n, h, w, c))
        if kind == "conv_infer":
            return dict(case=case, x=x, w=rnd(kh, kw, c, k) * math.sqrt(2.0 / (kh * kw * c)), bias=0.1 * rnd(k),
                        scale=1.0 + 0.1 * rnd(k))
        oh, ow = _conv_out(case)
        layer = layers.AMConv2D(c, k, (kh, kw), strides=case["stride"], padding=case["padding"].lower(), mant_mul_lut=lut,
                                deterministic=det).cuda()
        _fill([layer.kernel, layer.bias], gen, [kh * kw * c, 0])
        return dict(case=case, layer=layer, x=x.requires_grad_(not case["image"]), dy=1e-3 * rnd(n, oh, ow, k))
    if kind == "dense_train":
        layer = layers.denseam(case["width"], case["units"], mant_mul_lut=lut, deterministic=det).cuda()
        _fill([layer.kernel, layer.bias], gen, [case["width"], 0])
        return dict(case=case, layer=layer, x=rnd(case["rows"], case["width"]).requires_grad_(),
                    dy=1e-3 * rnd(case["rows"], case["units"]))
    b, h, s, d = case["n"], case["heads"], case["seq"], case["depth"]
    q, k, v = (rnd(b, h, s, d).requires_grad_() for _ in range(3))
    return dict(case=case, q=q, k=k, v=v, do=1e-3 * rnd(b, h, s, d), alpha=1.0 / math.sqrt(d))


def run(state):
    case = state["case"]
    kind, lut, det = case["kind"], _lut(case), case["det"]
    if kind == "mlp_infer":
        with torch.no_grad():
            return state["net"](state["x"])
    if kind == "lenet5_step":
        loss = state["trainer"].step(state["loss"])
        return [loss] + [p.detach() for p in state["net"].parameters()]
    if kind == "conv_infer":
        return ops.convam_bias_act(state["x"], state["w"], state["bias"], strides=case["stride"], padding=case["padding"],
                                   activation="relu", mant_mul_lut=lut, deterministic=det, scale=state["scale"])
    if kind in ("conv_train", "dense_train"):
        layer, x = state["layer"], state["x"]
        y = layer(x)
        wrt = ([x] if x.requires_grad else []) + [layer.kernel, layer.bias]
        return [y.detach(), *torch.autograd.grad(y, wrt, state["dy"])]
    q, k, v = state["q"], state["k"], state["v"]
    weights = torch.softmax(layers.ammatmul(q, k, lut, det, transpose_b=True, alpha=state["alpha"]), -1)
    o = layers.ammatmul(weights, v, lut, det)
    return [o.detach(), *torch.autograd.grad(o, (q, k, v), state["do"])]
