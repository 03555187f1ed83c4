"""The work that users of this package have it do, as measurable cases.

Two kinds of case, both through the package's public entry points:

* ``layer``: one ``DepthwiseOrientedConv1d`` module, called for inference (``forward``) or for
  training (forward, then the gradients of input, weight and bias through autograd);
* ``model``: a ``ConvNeXt1D`` classifier, called for inference, or for training (cross-entropy and
  all parameter gradients in one flat buffer, as a data-parallel step keeps them).

Angles of a layer: ``blocks`` (eight contiguous channel groups, as the models assign them), ``cycle``
(channel c has angle c mod 8, as the operator benchmark assigns them) or ``one`` (a single angle,
the module's own default form; ``turn`` counts it in steps of 22.5 degrees).
"""
import math

import torch
import torch.nn.functional as F

from oriented1d_b200 import DepthwiseOrientedConv1d
from oriented1d_b200.convnext1d import ConvNeXt1D

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
MODELS = {"tiny": ((3, 3, 9, 3), (96, 192, 384, 768)), "base": ((3, 3, 27, 3), (128, 256, 512, 1024))}
CLASSES = 1000


def _layer(name=None, N=1, H=14, W=14, C=384, K=31, stride=1, dtype="bf16", layout="nhwc", angles="blocks", turn=0,
           resid=False, train=True):
    c = dict(kind="layer", N=N, H=H, W=W, C=C, K=K, stride=stride, dtype=dtype, layout=layout, angles=angles, turn=turn,
             resid=resid, train=train)
    return c if name is None else dict(c, name=name)


def _model(name=None, variant="1d", size="tiny", batch=1, image=224, train=False):
    c = dict(kind="model", variant=variant, size=size, batch=batch, image=image, train=train)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # serving one image: the smallest call, a block's conv in the third stage
        _layer("layer-1x14x14x384-bf16-fwd", N=1, H=14, W=14, C=384, train=False),
        # a user's first training check: two images, first-stage map, fp32
        _layer("layer-2x56x56x96-fp32", N=2, H=56, W=56, C=96, dtype="fp32", angles="cycle"),
        # the stage shapes of the tiny classifier at the benchmark's batch
        _layer("stage1-128x56x56x96-fp32", N=128, H=56, W=56, C=96, dtype="fp32", angles="cycle"),
        _layer("stage2-128x28x28x192-bf16", N=128, H=28, W=28, C=192, angles="cycle"),
        _layer("stage4-128x7x7x768-bf16", N=128, H=7, W=7, C=768, angles="cycle"),
        # the second conv of a base 1D++ block, on the hidden tensor (27 of them in a training step)
        _layer("hidden-64x14x14x2048-bf16", N=64, H=14, W=14, C=2048, resid=True),
        # a layer inside an unchanged NCHW fp32 model, at the channel count of the published operator timings
        _layer("nchw-64x28x28x512-fp32", N=64, H=28, W=28, C=512, dtype="fp32", layout="nchw"),
        # the stem's first conv in training
        _layer("stem-64x224x224x64-s2-bf16", N=64, H=224, W=224, C=64, stride=2),
        # first stage of a detection backbone on a padded batch: large, ragged
        _layer("dense-2x200x333x96-bf16", N=2, H=200, W=333, C=96),
        # classifier inference: one image (latency) and a full batch
        _model("tiny-1d-infer-1", batch=1),
        _model("tiny-1d-infer-256", batch=256),
        # data-parallel training step of the base 1D++ classifier, per-GPU share
        _model("base-1dpp-train-64", variant="1dpp", size="base", batch=64, train=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    if rng.random() < 0.2:
        train = rng.random() < 0.5
        return _model(variant=rng.choice(["1d", "1dpp"]), size="tiny", batch=int(_log(rng, 1, 65 if train else 257)),
                      image=rng.choice([160, 192, 224, 256]), train=train)
    H = int(_log(rng, 7, 225))
    W = min(336, max(7, int(H * rng.uniform(0.75, 1.7))))
    C = 8 * int(_log(rng, 4, 257))                      # 32 .. 2048, a multiple of 8
    elements = _log(rng, 6e4, 3.8e7)
    N = min(256, max(1, int(elements / (H * W * C))))
    C = min(C, 8 * max(4, int(3.8e7 / (8 * N * H * W))))
    angles = rng.choice(["blocks", "blocks", "cycle", "one"])
    return _layer(N=N, H=H, W=W, C=C, K=rng.choice([7, 13, 15, 27, 31, 31, 31]), stride=2 if rng.random() < 0.15 else 1,
                  dtype=rng.choice(["bf16", "bf16", "fp32"]), layout=rng.choice(["nhwc", "nhwc", "nhwc", "nchw"]),
                  angles=angles, turn=rng.randrange(8) if angles == "one" else 0, resid=rng.random() < 0.3,
                  train=rng.random() < 0.7)


def _angles(case):
    C = case["C"]
    if case["angles"] == "blocks":
        return [math.pi * (((8 * (c + 1) - 1) // C) / 8) for c in range(C)]
    if case["angles"] == "cycle":
        return [math.pi * (c % 8) / 8 for c in range(C)]
    return math.pi * case["turn"] / 8


def _out_hw(case):
    return -(-case["H"] // case["stride"]), -(-case["W"] // case["stride"])


def _prepare_layer(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt, C, K = DTYPES[case["dtype"]], case["C"], case["K"]
    nhwc = case["layout"] == "nhwc"
    conv = DepthwiseOrientedConv1d(C, C, K, groups=C, stride=case["stride"], padding=K // 2, angle=_angles(case), nhwc=nhwc,
                                   resid=case["resid"], arbitrary_size=True).to("cuda", dt)

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g, dtype=torch.float32)

    def activation(h, w):
        return normal(*((case["N"], h, w, C) if nhwc else (case["N"], C, h, w)))

    with torch.no_grad():
        conv.weight.copy_(0.02 * normal(C, 1, 1, K))
        conv.bias.copy_(0.02 * normal(C))
    x = activation(case["H"], case["W"])
    if case["resid"]:                                   # the conv with the identity tap follows a GELU
        x = F.gelu(x)
    state = {"kind": "layer", "train": case["train"], "conv": conv, "x": x.to(dt)}
    if case["train"]:
        state["x"].requires_grad_(True)
        state["dy"] = activation(*_out_hw(case)).to(dt)
    else:
        conv.eval()
    return state


def _prepare_model(case, seed):
    depths, dims = MODELS[case["size"]]
    with torch.random.fork_rng(devices=[torch.cuda.current_device()]):
        torch.manual_seed(seed)
        with torch.device("cuda"):
            model = ConvNeXt1D(depths=depths, dims=dims, num_classes=CLASSES, variant=case["variant"],
                               drop_path_rate=0.0, layer_scale_init_value=1e-1)
        model = model.to("cuda", torch.bfloat16)
        x = torch.randn(case["batch"], 3, case["image"], case["image"], device="cuda").to(torch.bfloat16)
        labels = torch.randint(0, CLASSES, (case["batch"],), device="cuda")
    state = {"kind": "model", "train": case["train"], "model": model, "x": x}
    if not case["train"]:
        model.eval()
        return state
    params = [p for n, p in model.named_parameters() if not n.endswith("theta")]
    flat = torch.zeros(sum(p.numel() for p in params), dtype=torch.bfloat16, device="cuda")
    at = 0
    for p in params:
        p.grad = flat[at:at + p.numel()].view_as(p)
        at += p.numel()
    return dict(state, labels=labels, flat=flat)


def prepare(case, seed):
    return _prepare_layer(case, seed) if case["kind"] == "layer" else _prepare_model(case, seed)


def run(state):
    if state["kind"] == "layer":
        conv, x = state["conv"], state["x"]
        if not state["train"]:
            with torch.no_grad():
                return {"y": conv(x)}
        y = conv(x)
        dx, dw, db = torch.autograd.grad(y, (x, conv.weight, conv.bias), state["dy"])
        return {"y": y.detach(), "dx": dx, "dw": dw, "db": db}
    model = state["model"]
    if not state["train"]:
        with torch.no_grad():
            return {"logits": model(state["x"])}
    state["flat"].zero_()
    loss = F.cross_entropy(model(state["x"]).float(), state["labels"])
    loss.backward()
    return {"loss": loss.detach(), "gradients": state["flat"]}


def work(case):
    if case["kind"] == "layer":
        e = 4 if case["dtype"] == "fp32" else 2
        P, Q = _out_hw(case)
        x, y = case["N"] * case["H"] * case["W"] * case["C"], case["N"] * P * Q * case["C"]
        params = case["C"] * (case["K"] + 1)
        passes = 3 if case["train"] else 1              # output, input gradient, weight gradient
        return {"bytes": e * (x + y + params) * (2 if case["train"] else 1), "flops": 2 * passes * y * case["K"]}
    # a model: its matrix products and oriented convolutions; bytes: images, parameters and gradients
    depths, dims = MODELS[case["size"]]
    batch, side, pp = case["batch"], case["image"], case["variant"] == "1dpp"
    first = 15 if pp else 31                            # taps of the stem's and each block's first conv
    p = side * side // 16                               # pixels per image of the first stage
    flops = 2 * (16 * p * 3 * 64 + 5 * p * 64 * first + p * 64 * dims[0])
    params = 3 * 64 + 64 * dims[0] + CLASSES * dims[3]
    for i, (depth, d) in enumerate(zip(depths, dims)):
        block = 8 * d * d + d * first + (4 * d * 31 if pp else 0)
        flops += 2 * depth * p * block
        params += depth * block
        if i < 3:
            p //= 4
            flops += 2 * p * 4 * d * dims[i + 1]
            params += 4 * d * dims[i + 1]
    passes = 3 if case["train"] else 1
    flops = batch * (flops * passes + 2 * CLASSES * dims[3])
    return {"bytes": 2 * (batch * 3 * side * side + params * (2 if case["train"] else 1)), "flops": flops}


def tolerance(case):
    if case["kind"] == "model":                         # rounding to bf16 after every layer
        return {"rel": 2e-2, "max": 0.5}
    if case["dtype"] == "bf16":
        return {"rel": 5e-3, "max": 5e-2}
    # fp32 sums; the weight gradient adds up to 1e5 products in an order of the kernel's own
    return {"rel": 1e-5, "max": 2e-4}
