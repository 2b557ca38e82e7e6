"""The framework's workloads as timed cases: what its users run, through its public entry points.

Four kinds of case:

``forward``     ``ddf(x, cf, sf, k, d, s, combine)`` under ``no_grad``: inference with the operator.
``train``       the same with all three gradients, through autograd.
``layer_train`` a ``DDFPack`` layer's training step under autocast (float32 parameters, 2-byte
                activations), every parameter's gradient included.
``network``     ``ddf_{mul,add}_resnet50`` inference, channels_last, BatchNorm folded.

Ranges (``draw``): 1 to 128 samples, 16 to 512 channels, planes from 7 x 7 to 300 pixels a side --
half of them the square feature maps of a 224-pixel ImageNet network (56, 28, 14, 7), half of any
height and width, as detection, segmentation and multi-scale crops give them -- kernel 3 and 5,
dilation 1 and 2, stride 1 and 2, both combine modes, float32, float16 and bfloat16.
"""
from __future__ import annotations

import math

import torch

from ddfnet_b200 import DDFPack, ddf
from ddfnet_b200.resnet import MODELS, fold_batchnorm

_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
_BYTES = {"f32": 4, "f16": 2, "bf16": 2}

# No operator case reads more than this many input elements (the largest listed one's).
_MOST_ELEMENTS = 2 * 256 * 200 * 300
# Images of 224 x 224 in the largest network pass.
_MOST_IMAGES = 256


def _op(kind, dtype, b, c, h, w, k=3, d=1, s=1, combine="mul"):
    return {"kind": kind, "dtype": dtype, "b": b, "c": c, "h": h, "w": w, "k": k, "d": d, "s": s,
            "combine": combine}


def listed():
    return [
        # One image through a late stage of a deployed network: a call's latency is the cost.
        {"name": "forward_one_image", **_op("forward", "f16", 1, 256, 14, 14)},
        # The first stage of a 50-layer network at a batch of 128: its largest operator call.
        {"name": "forward_stage1_batch", **_op("forward", "bf16", 128, 64, 56, 56)},
        # The down-sampling layer of the last stage, 'add' filters: many small planes.
        {"name": "forward_downsample", **_op("forward", "f16", 128, 512, 14, 14, s=2, combine="add")},
        # A detector's stride-4 feature map of a two-image batch, float32.
        {"name": "forward_detector_map", **_op("forward", "f32", 2, 256, 200, 300)},
        # A segmentation head with a wide field of view (5 x 5, dilation 2) on crops of odd size.
        {"name": "forward_wide_odd_crop", **_op("forward", "bf16", 8, 96, 75, 101, k=5, d=2, combine="add")},
        # Training at full precision, the third stage before its down-sampling.
        {"name": "train_stage3_f32", **_op("train", "f32", 64, 256, 28, 28)},
        # Training with 5 x 5 filters, 2-byte types.
        {"name": "train_5x5_bf16", **_op("train", "bf16", 64, 256, 28, 28, k=5)},
        # Training a down-sampling layer.
        {"name": "train_downsample", **_op("train", "bf16", 64, 128, 56, 56, s=2, combine="add")},
        # Fine-tuning a detector: few images, a plane size that no network stage has.
        {"name": "train_odd_map", **_op("train", "f16", 4, 128, 50, 67)},
        # The last stage on a fine-tuning batch of two: a step made of launches.
        {"name": "train_small", **_op("train", "bf16", 2, 512, 7, 7)},
        # A layer of the third stage in a mixed-precision training step.
        {"name": "layer_train_amp", "kind": "layer_train", "dtype": "f16", "b": 64, "c": 256, "h": 14, "w": 14,
         "s": 1, "combine": "mul"},
        # Whole-network inference at the evaluation batch.
        {"name": "network_batch", "kind": "network", "dtype": "f16", "model": "ddf_mul_resnet50", "b": 256,
         "image": 224},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng):
    """Mostly multiples of 8, as networks have; a quarter of any number."""
    c = _log_int(rng, 16, 512)
    return c if rng.random() < 0.25 else max(16, (c + 4) // 8 * 8)


def _draw_op(rng, kind):
    k, d, s = rng.choice([(3, 1, 1)] * 5 + [(3, 1, 2)] * 2 + [(3, 2, 1), (5, 1, 1), (5, 2, 1)])
    if rng.random() < 0.5:
        h = w = rng.choice([7, 14, 28, 56] if s == 1 else [14, 28, 56])
        c = 64 * 56 // h if rng.random() < 0.5 else _channels(rng)
    else:
        h = _log_int(rng, 7, 300)
        w = min(300, max(7, int(h * math.exp(rng.uniform(-0.6, 0.6)))))
        c = _channels(rng)
    c = min(c, 512)
    # the wider field costs more per element: keep a drawn case below the largest listed one
    most = _MOST_ELEMENTS // (1 if kind == "forward" else 3) // (1 if k == 3 else 3)
    b = min(_log_int(rng, 1, 128), max(1, most // (c * h * w)))
    c = min(c, max(16, most // (b * h * w)))
    return _op(kind, rng.choice(["f32", "f16", "bf16"]), b, c, h, w, k, d, s, rng.choice(["mul", "add"]))


def draw(rng):
    kind = rng.choice(["forward"] * 5 + ["train"] * 5 + ["layer_train", "network"])
    if kind in ("forward", "train"):
        return _draw_op(rng, kind)
    if kind == "layer_train":
        c = rng.choice([64, 128, 256, 512])
        h = 64 * 56 // c + rng.choice([0, 0, 2, 6])
        s = rng.choice([1, 1, 2])
        return {"kind": kind, "dtype": rng.choice(["f16", "bf16"]), "b": _log_int(rng, 4, 96), "c": c,
                "h": h // s * s, "w": h // s * s, "s": s, "combine": rng.choice(["mul", "add"])}
    image = rng.choice([160, 192, 224, 224, 256, 288])
    b = min(_log_int(rng, 1, _MOST_IMAGES), _MOST_IMAGES * 224 * 224 // (image * image))
    return {"kind": kind, "dtype": rng.choice(["f16", "bf16"]),
            "model": rng.choice(["ddf_mul_resnet50", "ddf_add_resnet50"]), "b": b, "image": image}


def _op_inputs(case, seed):
    """Activations after a ReLU; filters of a FilterNorm (zero mean, std 1 / k); unit upstream gradient."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    b, c, h, w, k, s = (case[n] for n in ("b", "c", "h", "w", "k", "s"))

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)

    x = normal(b, c, h, w).relu_().to(dt)
    cf = normal(b, c, k, k).div_(k).to(dt)
    sf = normal(b, k * k, h // s, w // s).div_(k).to(dt)
    state = {"case": case, "x": x, "cf": cf, "sf": sf,
             "args": (k, case["d"], s, case["combine"])}
    if case["kind"] == "train":
        for t in (x, cf, sf):
            t.requires_grad_()
        state["go"] = normal(b, c, h // s, w // s).to(dt)
    return state


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forward", "train"):
        return _op_inputs(case, seed)
    dt = _DTYPES[case["dtype"]]
    torch.manual_seed(seed)
    if kind == "layer_train":
        with torch.device("cuda"):
            layer = DDFPack(case["c"], kernel_size=3, stride=case["s"], kernel_combine=case["combine"]).train()
            x = torch.randn(case["b"], case["c"], case["h"], case["w"]).relu_().to(dt).requires_grad_()
            go = torch.randn(case["b"], case["c"], case["h"] // case["s"], case["w"] // case["s"])
        return {"case": case, "layer": layer, "x": x, "go": go, "params": list(layer.parameters())}
    with torch.device("cuda"):
        model = MODELS[case["model"]]().eval()
        with torch.no_grad():
            for m in model.modules():  # statistics of a network that has seen data
                if isinstance(m, torch.nn.BatchNorm2d):
                    m.running_mean.normal_(0, 0.1)
                    m.running_var.uniform_(0.5, 2)
            for block in model.modules():  # residual branches that leave the shortcut's scale alone
                if hasattr(block, "bn3"):
                    block.bn3.weight.fill_(0.5)
            fold_batchnorm(model, fuse_activations=True)
            model = model.to(dt).to(memory_format=torch.channels_last)
        x = torch.randn(case["b"], 3, case["image"], case["image"]).to(dt)
    return {"case": case, "model": model, "x": x.contiguous(memory_format=torch.channels_last)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "forward":
        with torch.no_grad():
            return ddf(state["x"], state["cf"], state["sf"], *state["args"])
    if kind == "train":
        x, cf, sf = state["x"], state["cf"], state["sf"]
        out = ddf(x, cf, sf, *state["args"])
        gx, gcf, gsf = torch.autograd.grad(out, (x, cf, sf), state["go"])
        return {"out": out, "gx": gx, "gcf": gcf, "gsf": gsf}
    if kind == "layer_train":
        with torch.autocast("cuda", dtype=_DTYPES[case["dtype"]]):
            out = state["layer"](state["x"])
        # float32 filter gains make the layer's output, and so its gradient, float32
        grads = torch.autograd.grad(out, [state["x"], *state["params"]], state["go"])
        return [out, *grads]
    with torch.no_grad():
        return state["model"](state["x"])


def _op_work(case, es):
    b, c, h, w, k, s = (case[n] for n in ("b", "c", "h", "w", "k", "s"))
    x, cf, sf, out = b * c * h * w, b * c * k * k, b * k * k * (h // s) * (w // s), b * c * (h // s) * (w // s)
    taps = out * k * k
    if case["kind"] == "forward":
        return {"bytes": es * (x + cf + sf + out), "flops": 3 * taps}
    # x, filters and upstream gradient read once; output and three gradients written once
    return {"bytes": es * 2 * (x + cf + sf + out), "flops": (3 + 3 + 5) * taps}


def _network_flops(case):
    """Multiply-adds (counted twice) of the convolutions and the dynamic filters of a 50-layer network."""
    side = case["image"] // 2
    flops = 2 * side * side * 64 * 3 * 49
    side //= 2
    cin = 64
    for planes, blocks, stride in ((64, 3, 1), (128, 4, 2), (256, 6, 2), (512, 3, 2)):
        for i in range(blocks):
            s = stride if i == 0 else 1
            out = side // s
            flops += 2 * side * side * cin * planes          # 1 x 1 in
            flops += 2 * out * out * planes * 9              # spatial branch
            flops += 3 * out * out * planes * 9              # dynamic filter
            flops += 2 * out * out * planes * 4 * planes     # 1 x 1 out
            if i == 0:
                flops += 2 * out * out * cin * 4 * planes    # shortcut
            side, cin = out, 4 * planes
    return case["b"] * (flops + 2 * 2048 * 1000)


def work(case):
    kind = case["kind"]
    es = _BYTES[case["dtype"]]
    if kind in ("forward", "train"):
        return _op_work(case, es)
    if kind == "layer_train":
        b, c, h, w, s = (case[n] for n in ("b", "c", "h", "w", "s"))
        mid = int(c * 0.2)
        x, out = b * c * h * w, b * c * (h // s) * (w // s)
        params = 9 * c + 9 + mid * c + mid + 9 * c * mid + 9 * c + 9 * c
        # activations read and their gradients written once, parameters likewise in float32
        conv = 2 * 9 * out + 2 * b * mid * c * 10
        return {"bytes": es * 2 * (x + out) + 4 * 2 * params, "flops": 11 * 9 * out + 3 * conv}
    params = 16.8e6
    return {"bytes": es * (case["b"] * (3 * case["image"] ** 2 + 1000) + params), "flops": _network_flops(case)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("forward", "train"):
        # float32 sums in another order; one rounding to the 2-byte type on each side
        return {"f32": {"rel": 1e-5, "max": 2e-4},
                "f16": {"rel": 1e-3, "max": 4e-3},
                "bf16": {"rel": 5e-3, "max": 2e-2}}[case["dtype"]]
    # chains of roundings to the 2-byte type: about ten in the layer, about fifty in the network
    return {"rel": 1e-2 if case["dtype"] == "f16" else 2.5e-2}
