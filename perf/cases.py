"""What this framework is timed on: the calls a training program makes, over the range it makes them.

A training step with compressed activations consists of few kinds of work, and there is a family
of cases for each of them:

``codec``     one activation through ``ops.quantize_activation`` / ``dequantize_activation``: the pair
              every layer that saves an activation goes through once per step.  ``level`` "L3" is the
              default (2 bits on average, adaptive per sample), "L2" the uniform 4-bit level, and
              ``bits`` overrides the average width.
``bn``        forward and backward of a ``QBatchNorm2d`` in training mode;
``relu_pool`` forward and backward of ``QReLU`` followed by ``QMaxPool2d``, the stem of most networks;
``conv``      forward and backward of a 3x3 ``QConv2d`` followed by ``QReLU``;
``head``      forward and backward of a classifier head, ``QLinear`` - ``QReLU`` - ``QDropout`` - ``QLinear``;
``block``     forward and backward of a residual bottleneck block converted by ``QModule``;
``net``       forward and backward of a small convolutional classifier converted by ``QModule``.

``prepare`` makes what a program holds before the step: layers, activations, upstream gradients.
``run`` makes one step.  The rounding noise and the dropout masks come from torch's CUDA generator,
which every step seeds, as a program does that wants its steps to be reproducible.
"""
import math

import torch
import torch.nn as nn

import actnn_b200 as actnn
from actnn_b200 import ops
from actnn_b200.conf import QuantizationConfig, config

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
BYTES = {"f16": 2, "bf16": 2, "f32": 4}
GROUP = 256                                    # elements that share one (scale, min), config.group_size
MOST_ELEMENTS = 512 * 256 * 28 * 28            # the largest single activation of the listed cases


def listed():
    return [
        # the smallest call: a few samples of a narrow map whose samples are not whole groups (3136 = 12.25 x 256)
        dict(name="codec_l3_small_f16", kind="codec", level="L3", bits=0, n=8, c=16, h=14, w=14, dtype="f16"),
        # an ordinary ragged one, as detection and segmentation inputs give: odd map, 918.75 groups a sample
        dict(name="codec_l3_ragged_f16", kind="codec", level="L3", bits=0, n=100, c=192, h=35, w=35, dtype="f16"),
        # the largest: the activation of the benchmark
        dict(name="codec_l3_bf16", kind="codec", level="L3", bits=0, n=512, c=256, h=28, w=28, dtype="bf16"),
        # the uniform level with its 4 bits, on a middle layer of a ResNet at batch 256
        dict(name="codec_l2_4bit_f16", kind="codec", level="L2", bits=0, n=256, c=256, h=28, w=28, dtype="f16"),
        # uniform 2 bits of a float32 activation (training without autocast)
        dict(name="codec_2bit_f32", kind="codec", level="L2", bits=2, n=64, c=64, h=56, w=56, dtype="f32"),
        # batch norm of an early layer (large maps) and of a late one (14x14 maps)
        dict(name="bn_l3_56_f16", kind="bn", level="L3", n=256, c=64, h=56, w=56, dtype="f16"),
        dict(name="bn_l3_14_f16", kind="bn", level="L3", n=128, c=256, h=14, w=14, dtype="f16"),
        # the stem of a ResNet: ReLU, then 3x3 / 2 max pooling of 112x112 maps
        dict(name="relu_pool_f16", kind="relu_pool", level="L3", n=128, c=64, h=112, w=112, k=3, dtype="f16"),
        # a 3x3 convolution with its ReLU
        dict(name="conv_relu_f16", kind="conv", level="L3", n=256, c=256, h=28, w=28, dtype="f16"),
        # a classifier head at batch 256 under autocast
        dict(name="head_f16", kind="head", level="L3", n=256, c=2048, hidden=4096, out=1000, dtype="f16"),
        # a bottleneck block of the second stage of a ResNet-50 at batch 256 under autocast
        dict(name="block_l3_f16", kind="block", level="L3", n=256, c=512, mid=128, h=28, w=28, dtype="f16"),
        # a small classifier of 32x32 images in float32: many short kernels, paced by launches and the host
        dict(name="net_l3_f32", kind="net", level="L3", n=256, c=16, h=32, w=32, out=100, dtype="f32"),
    ]


def _size(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm, odd as often as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["codec", "codec", "codec", "bn", "bn", "relu_pool", "conv", "head", "block", "net"])
    dtype = rng.choice(["f16", "f16", "bf16", "f32"])
    level = rng.choice(["L3", "L3", "L2"])
    if kind == "codec":
        c, hw, n = _size(rng, 3, 512), _size(rng, 5, 64), _size(rng, 4, 512)
        n = max(1, min(n, MOST_ELEMENTS // (c * hw * hw * (BYTES[dtype] // 2))))
        bits = rng.choice([0, 0, 0, 2, 3]) if level == "L3" else rng.choice([0, 0, 1, 2, 8])
        return dict(kind=kind, level=level, bits=bits, n=n, c=c, h=hw, w=max(1, hw - rng.choice([0, 0, 1, 3])),
                    dtype=dtype)
    if kind == "bn":
        c, hw, n = _size(rng, 8, 512), _size(rng, 5, 64), _size(rng, 8, 256)
        n = max(2, min(n, 256 * 64 * 56 * 56 // (c * hw * hw * (BYTES[dtype] // 2))))
        return dict(kind=kind, level=level, n=n, c=c, h=hw, w=hw, dtype=dtype)
    if kind == "relu_pool":
        c, hw, n = _size(rng, 8, 128), _size(rng, 8, 128), _size(rng, 4, 256)
        n = max(1, min(n, 128 * 64 * 112 * 112 // (c * hw * hw * (BYTES[dtype] // 2))))
        return dict(kind=kind, level=level, n=n, c=c, h=hw, w=hw, k=rng.choice([2, 3, 3]), dtype=dtype)
    dtype = rng.choice(["f16", "bf16"])
    if kind == "conv":
        c, hw, n = 8 * _size(rng, 2, 32), _size(rng, 7, 56), _size(rng, 16, 256)
        n = max(1, min(n, 256 * 256 * 28 * 28 // (c * hw * hw)))
        return dict(kind=kind, level=level, n=n, c=c, h=hw, w=hw, dtype=dtype)
    if kind == "head":
        return dict(kind=kind, level=level, n=_size(rng, 16, 512), c=8 * _size(rng, 32, 256), hidden=8 * _size(rng, 32, 512),
                    out=_size(rng, 10, 1000), dtype=dtype)
    if kind == "block":
        mid, hw, n = 8 * _size(rng, 4, 32), _size(rng, 7, 56), _size(rng, 128, 256)
        n = max(8, min(n, 256 * 128 * 28 * 28 // (mid * hw * hw)))
        return dict(kind=kind, level="L2" if n < 128 else level, n=n, c=4 * mid, mid=mid, h=hw, w=hw, dtype="f16")
    hw = 4 * _size(rng, 6, 12)
    return dict(kind="net", level=level, n=_size(rng, 128, 256), c=8 * _size(rng, 1, 4), h=hw, w=hw,
                out=_size(rng, 10, 200), dtype="f32")


# ------------------------------------------------------------------------------------- models
class _Bottleneck(nn.Module):
    """From one block's sum to the next one's: the ReLU that closes a block, then the next block."""

    def __init__(self, c, mid):
        super().__init__()
        self.conv1, self.bn1 = nn.Conv2d(c, mid, 1, bias=False), nn.BatchNorm2d(mid)
        self.conv2, self.bn2 = nn.Conv2d(mid, mid, 3, padding=1, bias=False), nn.BatchNorm2d(mid)
        self.conv3, self.bn3 = nn.Conv2d(mid, c, 1, bias=False), nn.BatchNorm2d(c)
        self.relu, self.relu1, self.relu2 = nn.ReLU(), nn.ReLU(), nn.ReLU()

    def forward(self, x):
        x = self.relu(x)
        y = self.relu1(self.bn1(self.conv1(x)))
        y = self.relu2(self.bn2(self.conv2(y)))
        return self.bn3(self.conv3(y)) + x


def _classifier(c, out):
    return nn.Sequential(
        nn.Conv2d(3, c, 3, padding=1, bias=False), nn.BatchNorm2d(c), nn.ReLU(),
        nn.Conv2d(c, 2 * c, 3, padding=1, bias=False), nn.BatchNorm2d(2 * c), nn.ReLU(), nn.MaxPool2d(2),
        nn.Conv2d(2 * c, 4 * c, 3, padding=1, bias=False), nn.BatchNorm2d(4 * c), nn.ReLU(), nn.MaxPool2d(2),
        nn.AdaptiveAvgPool2d(1), nn.Flatten(), nn.Linear(4 * c, out))


def _configure(case):
    """The settings a program makes at its start, from the defaults."""
    config.__dict__.update(QuantizationConfig().__dict__)
    actnn.set_optimization_level(case["level"])
    if case.get("bits"):
        config.activation_compression_bits = [case["bits"]] * len(config.activation_compression_bits)
    # the layers register themselves in process-wide lists, of which a program has one pair; several
    # independent models live in this process, each with its own
    actnn.QScheme.layers, actnn.QBNScheme.layers = [], []
    actnn.QScheme.prev_layer = None


def _made(state, **more):
    state.update(registry=(actnn.QScheme.layers, actnn.QBNScheme.layers), **more)
    return state


def prepare(case, seed):
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    torch.cuda.init()
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    torch.manual_seed(seed)                                    # layer initialisation
    rng = torch.cuda.default_generators[torch.cuda.current_device()]
    _configure(case)

    def randn(*shape, scale=1.0, to=dt):
        return (torch.randn(shape, device=dev, generator=gen) * scale).to(to)

    state = dict(kind=kind, seed=seed, rng=rng)
    n, c = case["n"], case["c"]
    with torch.device(dev):
        if kind == "codec":
            # outputs of a ReLU whose samples have different ranges
            spread = torch.exp(0.5 * torch.randn(n, 1, 1, 1, device=dev, generator=gen))
            x = (torch.relu(torch.randn(n, c, case["h"], case["w"], device=dev, generator=gen)) * spread).to(dt)
            scheme = actnn.QConv2d(c, 1, 3, padding=1).scheme
            if scheme is not None:                             # as after the first backward pass
                scheme.set_scale(randn(n, 64, scale=1e-2))
            return _made(state, x=x, scheme=scheme)
        if kind == "bn":
            layer = actnn.QBatchNorm2d(c)
            shift = torch.linspace(-1.0, 1.0, c, device=dev).view(1, c, 1, 1)
            x = (torch.randn(n, c, case["h"], case["w"], device=dev, generator=gen) * 1.5 + shift).to(dt)
            with torch.no_grad():
                layer.weight.uniform_(0.5, 1.5, generator=gen)
                layer.bias.normal_(0.0, 0.2, generator=gen)
            gy = randn(n, c, case["h"], case["w"], scale=1e-2)
            return _made(state, layer=layer, x=x.requires_grad_(), gy=gy)
        if kind == "relu_pool":
            k = case["k"]
            layer = nn.Sequential(actnn.QReLU(), actnn.QMaxPool2d(k, 2, 1 if k == 3 else 0))
            x = randn(n, c, case["h"], case["w"]).requires_grad_()
            ho = (case["h"] + (2 if k == 3 else 0) - k) // 2 + 1
            wo = (case["w"] + (2 if k == 3 else 0) - k) // 2 + 1
            return _made(state, layer=layer, x=x, gy=randn(n, c, ho, wo, scale=1e-2))
        if kind == "conv":
            conv = actnn.QConv2d(c, c, 3, padding=1, bias=False).to(dt)
            layer = nn.Sequential(conv, actnn.QReLU())
            with torch.no_grad():
                nn.init.kaiming_normal_(conv.weight, generator=gen)
            x = randn(n, c, case["h"], case["w"]).requires_grad_()
            return _made(state, layer=layer, x=x, gy=randn(n, c, case["h"], case["w"], scale=1e-2))
        if kind == "head":
            layer = nn.Sequential(actnn.QLinear(c, case["hidden"]), actnn.QReLU(), actnn.QDropout(0.5),
                                  actnn.QLinear(case["hidden"], case["out"]))
            x = torch.relu(randn(n, c)).requires_grad_()
            return _made(state, layer=layer, x=x, gy=randn(n, case["out"], scale=1e-2), autocast=dt)
        if kind == "block":
            layer = actnn.QModule(_Bottleneck(c, case["mid"]))
            x = randn(n, c, case["h"], case["w"]).requires_grad_()
            return _made(state, layer=layer.train(), x=x, gy=randn(n, c, case["h"], case["w"], scale=1e-2), autocast=dt)
        layer = actnn.QModule(_classifier(c, case["out"]))
        labels = torch.randint(case["out"], (n,), device=dev, generator=gen)
        return _made(state, layer=layer.train(), x=randn(n, 3, case["h"], case["w"]), labels=labels)


# ------------------------------------------------------------------------------------- one step
def run(state):
    actnn.QScheme.layers, actnn.QBNScheme.layers = state["registry"]
    state["rng"].manual_seed(state["seed"])
    x = state["x"]
    if state["kind"] == "codec":
        quantized = ops.quantize_activation(x, state["scheme"])
        restored = ops.dequantize_activation(quantized, x.shape, x.dtype)
        packed, bits, scale, minimum = quantized
        return {"packed": packed, "bits": bits, "scale": scale, "min": minimum, "restored": restored}
    layer = state["layer"]
    wanted = list(layer.parameters()) + ([x] if x.requires_grad else [])
    if "autocast" in state:
        with torch.autocast("cuda", dtype=state["autocast"]):
            y = layer(x)
    else:
        y = layer(x)
    if state["kind"] == "net":
        loss = nn.functional.cross_entropy(y, state["labels"])
        return {"logits": y, "loss": loss, "grads": torch.autograd.grad(loss, wanted)}
    out = {"y": y, "grads": torch.autograd.grad(y, wanted, state["gy"])}
    if state["kind"] == "bn":
        out["running_mean"], out["running_var"] = layer.running_mean, layer.running_var
    return out


# ------------------------------------------------------------------------------------- what a pass cannot do without
def _saved_bytes(case, elements, samples):
    """Bytes of a compressed activation: codes, and a scale and a minimum (2 bytes each) per group."""
    bits = case.get("bits") or {"L3": 2, "L2": 4}[case["level"]]
    groups = samples * -(-(elements // samples) // GROUP)
    return elements * bits / 8 + groups * 4


def work(case):
    kind, s, n, c = case["kind"], BYTES[case["dtype"]], case["n"], case["c"]
    if kind == "head":
        hid, out = case["hidden"], case["out"]
        macs = n * hid * (c + out)
        data = (2 * n * c + 4 * n * hid + 2 * n * out) * s + 2 * 4 * hid * (c + out)     # weights and their gradients: float32
        saved = _saved_bytes(case, n * c, n) + _saved_bytes(case, n * hid, n) + 2 * n * hid / 8
        return {"bytes": data + 2 * saved, "flops": 6 * macs}
    h, w = case["h"], case["w"]
    e = n * c * h * w
    if kind == "codec":
        return {"bytes": 2 * (e * s + _saved_bytes(case, e, n)), "flops": 12 * e}
    if kind == "bn":
        return {"bytes": 4 * e * s + 2 * _saved_bytes(case, e, n), "flops": 24 * e}
    if kind == "relu_pool":
        o = e / 4
        return {"bytes": 4 * e * s + 2 * e / 8 + 2 * o * (s + 1), "flops": (case["k"] ** 2 + 2) * o + 2 * e}
    if kind == "conv":
        data = 4 * e * s + 2 * e / 8 + 2 * 9 * c * c * s
        return {"bytes": data + 2 * _saved_bytes(case, e, n), "flops": 6 * 9 * e * c}
    if kind == "block":
        mid, m = case["mid"], n * case["mid"] * h * w
        # convolutions read and write their maps, the batch norms and ReLUs once more each; both directions
        data = (2 * (e + m + m + m + m + e) + 2 * (4 * m + 2 * e) + 2 * (4 * m + 3 * e)) * s
        saved = 2 * (_saved_bytes(case, e, n) * 2 + _saved_bytes(case, m, n) * 4) + 2 * (2 * m + e) / 8
        return {"bytes": data + saved, "flops": 6 * (2 * m * c + 9 * m * mid)}
    p = n * h * w
    maps = [p * c, p * 2 * c, p // 4 * 4 * c]
    macs = p * 27 * c + p * 9 * c * 2 * c + p // 4 * 9 * 2 * c * 4 * c + n * 4 * c * case["out"]
    data = 8 * 2 * sum(maps) * s + (p * 3 * s)
    saved = sum(2 * _saved_bytes(case, m, n) for m in maps) * 2
    return {"bytes": data + saved, "flops": 6 * macs}


def tolerance(case):
    """About four times what changes when the sums of the batch-norm statistics are taken in another
    order (ATen's kernels in place of this package's), measured over listed and drawn cases."""
    kind, dt = case["kind"], case["dtype"]
    if kind == "codec":
        return "exact"                     # codes, packed words and decoded values are defined to the bit, given the noise
    if kind == "relu_pool":
        # selections are exact; gradients of overlapping windows are summed in float32 and rounded once
        return {"rel": 1e-4, "max": 1e-2} if dt != "bf16" else {"rel": 1e-3, "max": 1e-2}
    if kind == "bn":
        # a few results round the other way: a unit in the last place each
        return {"f16": {"rel": 5e-5, "max": 4e-3}, "bf16": {"rel": 1e-4, "max": 3e-2}, "f32": {"rel": 2e-6, "max": 1e-5}}[dt]
    if kind in ("conv", "head"):
        return {"rel": 2e-3, "max": 5e-2} if dt == "f16" else {"rel": 1.2e-2, "max": 0.3}
    # several layers: such a unit moves later roundings, some 2-bit codes with them, and a few ReLU masks
    return {"rel": 2.5e-2, "max": 0.9 if kind == "block" else 0.25}
