"""Performance cases: calls of the public modules as a program makes them, over the sizes they meet.

A case names a module, its constructor arguments, the input's size and whether the call is a training step (forward
and all gradients, through autograd) or an inference forward.  `listed()` has the ones that stand for a use each,
`draw()` others of the same ranges.
"""
from __future__ import annotations

import math

import torch

import deform_conv3d_pytorch_op_b200 as dcn

# op: deform = ConvOffset2d / ConvOffset3d (offsets are an input), plain = Conv2d / Conv3d,
#     layer = DeformLayer2d / DeformLayer3d (offset-producing convolution and deformable convolution in one call)
# size, k, stride, pad, dil: by axis, as text; g: groups; dg: deformable groups; offset_std: in input pixels
_DEFAULTS = {"op": "deform", "dtype": "float32", "precision": "exact", "train": True, "stride": "1", "pad": "1",
             "dil": "1", "g": 1, "dg": 1, "bias": False, "channels_last": False, "oob": True, "offset_std": 2.0}


def _case(**kw):
    return dict(_DEFAULTS, **kw)


def listed():
    return [
        # The call of a gradient check or a unit test: a few hundred values, all launches and host work.
        _case(name="3d tiny step", n=2, c=2, o=4, size="7x7x7", k="3", stride="2", pad="2", dil="2", g=2, bias=True,
              offset_std=0.6),
        # Benchmark configuration 1: a small 2-D layer in the default fp32 arithmetic, launch-bound.
        _case(name="2d small step", n=2, c=16, o=32, size="32x32", k="3"),
        # A mid-network 2-D layer of an unmodified fp32 program (default precision), odd sizes, a ragged batch.
        _case(name="2d fp32 step", n=6, c=96, o=96, size="33x45", k="3", dg=2, bias=True),
        # The double-precision package: used for gradient checks and reference runs.
        _case(name="2d fp64 step", n=2, c=32, o=32, size="28x28", k="3", dtype="float64", bias=True),
        # Benchmark configuration 2: a ResNet stage of 256 channels at 56x56, training on the tensor cores.
        _case(name="2d bf16 step", n=32, c=256, o=256, size="56x56", k="3", precision="bf16", dg=4, offset_std=3.0),
        # A detection network's high-resolution level: planes of an odd size, more than shared memory holds.
        _case(name="2d bf16 large plane step", n=2, c=128, o=128, size="101x151", k="3", precision="bf16", dg=2,
              bias=True),
        # Serving one image: forward only, batch 1, a ragged feature map.
        _case(name="2d bf16 inference", n=1, c=256, o=256, size="50x76", k="3", precision="bf16", train=False,
              bias=True),
        # Benchmark configuration 3: video features at full resolution; the largest work here.
        _case(name="3d bf16 step", n=8, c=64, o=64, size="16x56x56", k="3", precision="bf16", offset_std=1.5),
        # Benchmark configuration 4: groups, deformable groups, stride and dilation, fp32.
        _case(name="3d fp32 grouped step", n=16, c=128, o=256, size="8x28x28", k="3", stride="1x2x2", pad="2", dil="2",
              g=4, dg=8),
        # A late layer of the video network (configuration 5), inside a channels-last model; few positions.
        _case(name="3d bf16 channels-last step", n=64, c=256, o=256, size="2x7x7", k="3", precision="bf16", dg=4,
              channels_last=True, oob=False, offset_std=0.3),
        # The two-convolution pattern of the model scripts as one layer, training on the tensor cores.
        _case(name="2d bf16 layer step", op="layer", n=8, c=128, o=128, size="28x28", k="3", precision="bf16", dg=4,
              bias=True, offset_std=0.6),
        # The plain convolution package in its default arithmetic, a downsampling layer.
        _case(name="2d plain fp32 step", op="plain", n=8, c=64, o=128, size="56x56", k="3", stride="2", bias=True),
    ]


def _axes(case):
    size = [int(v) for v in case["size"].split("x")]

    def each(text):
        v = [int(t) for t in text.split("x")]
        return v * len(size) if len(v) == 1 else v

    k, stride, pad, dil = (each(case[f]) for f in ("k", "stride", "pad", "dil"))
    # the deformable operators' size rule leaves dilation out
    reach = [d * (m - 1) + 1 if case["op"] == "plain" else m for m, d in zip(k, dil)]
    out = [(s + 2 * p - r) // t + 1 for s, p, r, t in zip(size, pad, reach, stride)]
    return size, k, stride, pad, dil, out


def _counts(case):
    size, k, _, _, _, out = _axes(case)
    kv = math.prod(k)
    n, c, o = case["n"], case["c"], case["o"]
    return {"x": n * c * math.prod(size), "y": n * o * math.prod(out), "w": o * (c // case["g"]) * kv,
            "off": n * case["dg"] * kv * len(k) * math.prod(out), "ow": case["dg"] * kv * len(k) * c * kv,
            "positions": n * math.prod(out), "kv": kv, "corners": n * c * kv * math.prod(out) * 2 ** len(k)}


def _contraction(case):
    """Floating-point operations of one contraction pass."""
    t = _counts(case)
    f = 2.0 * t["positions"] * case["o"] * (case["c"] // case["g"]) * t["kv"]
    return f + (2.0 * t["positions"] * t["ow"] if case["op"] == "layer" else 0.0)


def work(case):
    """Each input read once and each output written once; one contraction forward, two backward."""
    t = _counts(case)
    item = 8 if case["dtype"] == "float64" else 4
    weights = t["w"] + (t["ow"] if case["op"] == "layer" else 0)
    offsets = t["off"] if case["op"] == "deform" else 0
    values = t["x"] + weights + offsets + t["y"]
    if case["train"]:
        values += t["y"] + t["x"] + weights + offsets        # grad_output in, the gradients out
    return {"bytes": item * values, "flops": _contraction(case) * (3 if case["train"] else 1)}


def tolerance(case):
    if case["precision"] == "bf16":
        return {"rel": 1e-2}             # operands rounded to bf16, fp32 sums
    return {"rel": 1e-12} if case["dtype"] == "float64" else {"rel": 1e-5}


def prepare(case, seed):
    size, k, stride, pad, dil, out = _axes(case)
    nd = len(size)
    dtype = getattr(torch, case["dtype"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    layout = {"memory_format": torch.channels_last if nd == 2 else torch.channels_last_3d} if case["channels_last"] else {}

    def normal(*shape, std=1.0):
        return torch.randn(shape, generator=g, device="cuda", dtype=dtype) * std

    cls = getattr(dcn, {"deform": "ConvOffset", "plain": "Conv", "layer": "DeformLayer"}[case["op"]] + "%dd" % nd)
    args = dict(stride=tuple(stride), padding=tuple(pad), dilation=tuple(dil), groups=case["g"], bias=case["bias"],
                precision=case["precision"], device="cuda", dtype=dtype)
    if case["op"] != "plain":
        args.update(channel_per_group=case["c"] // case["dg"], oob_offset_grad=case["oob"])
    m = cls(case["c"], case["o"], tuple(k), **args)
    kv = math.prod(k)
    with torch.no_grad():                 # trained-looking weights, from the seed
        for name, p in m.named_parameters():
            std = (2.0 / (case["o"] * kv)) ** 0.5 if p.dim() > 1 else 0.1
            if name.startswith("conv_offset."):
                std = case["offset_std"] / (case["c"] * kv / 3.0) ** 0.5 if p.dim() > 1 else 0.05
            p.copy_(normal(*p.shape, std=std))
    train = case["train"]
    x = torch.rand((case["n"], case["c"], *size), generator=g, device="cuda", dtype=dtype) * 2 - 1
    x = x.contiguous(**layout).requires_grad_(train)
    inputs = [x]
    if case["op"] == "deform":
        off = normal(case["n"], m.offset_channels, *out, std=case["offset_std"])
        inputs.append(off.requires_grad_(train))
    dy = normal(case["n"], case["o"], *out).contiguous(**layout) if train else None
    m.requires_grad_(train)
    return {"module": m, "inputs": inputs, "grads_of": inputs + list(m.parameters()), "dy": dy}


def run(state):
    if state["dy"] is None:
        with torch.no_grad():
            return state["module"](*state["inputs"])
    y = state["module"](*state["inputs"])
    return (y,) + torch.autograd.grad(y, state["grads_of"], state["dy"])


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# By kind of use: share of the draws; ranges of batch, channels, each spatial axis; channels come in multiples of
# `step` per group; the most contraction operations and corner values of a pass.
_KINDS = [
    (3, dict(nd=2, precision="exact", n=(1, 8), c=(2, 128), hw=(5, 64), step=1, flops=6e9, corners=1e8)),
    (2, dict(nd=3, precision="exact", n=(1, 8), c=(2, 128), hw=(4, 32), l=(2, 9), step=1, flops=16e9, corners=4e8)),
    (1, dict(nd=2, precision="exact", n=(1, 4), c=(2, 48), hw=(5, 32), step=1, flops=1e9, corners=3e7, dtype="float64")),
    (4, dict(nd=2, precision="bf16", n=(1, 32), c=(16, 512), hw=(7, 160), step=8, flops=118e9, corners=9e8)),
    (3, dict(nd=3, precision="bf16", n=(1, 64), c=(16, 512), hw=(4, 57), l=(1, 16), step=8, flops=88e9, corners=5e9)),
    (1, dict(nd=2, op="layer", precision="bf16", n=(1, 16), c=(16, 256), hw=(7, 56), step=8, flops=60e9, corners=4e8)),
    (1, dict(nd=2, op="plain", precision="exact", n=(1, 16), c=(3, 128), hw=(7, 64), step=1, flops=6e9, corners=1e8)),
]


def draw(rng):
    kind = rng.choices([k for _, k in _KINDS], [s for s, _ in _KINDS])[0]
    while True:
        g = rng.choice((1, 1, 1, 2, 4))
        dg = rng.choice((1, 1, 2, 4, 8)) if kind.get("op") != "plain" else 1
        unit = math.lcm(g, dg) * kind["step"]
        c = max(1, _log(rng, *kind["c"]) // unit) * unit
        o = max(1, round(c * rng.choice((0.5, 1, 1, 2)) / (g * kind["step"]))) * g * kind["step"]
        hw = _log(rng, *kind["hw"])
        size = [hw, max(kind["hw"][0], min(kind["hw"][1], round(hw * rng.uniform(0.7, 1.5))))]
        if kind["nd"] == 3:
            size.insert(0, _log(rng, *kind["l"]))
        k = rng.choice((3, 3, 3, 3, 1))
        dil = rng.choice((1, 1, 1, 2)) if k > 1 else 1
        cl = kind["precision"] == "bf16" and kind.get("op") != "layer" and rng.random() < 0.25
        case = _case(n=_log(rng, *kind["n"]), c=c, o=o, size="x".join(str(s) for s in size), k=str(k),
                     stride=str(rng.choice((1, 1, 1, 2))), pad=str(dil if k > 1 else 0), dil=str(dil), g=g, dg=dg,
                     bias=rng.random() < 0.5, precision=kind["precision"], dtype=kind.get("dtype", "float32"),
                     op=kind.get("op", "deform"), train=rng.random() < 0.75, channels_last=cl,
                     oob=kind["nd"] == 2 or rng.random() < 0.5, offset_std=round(rng.uniform(0.3, 3.0), 2))
        if case["op"] == "layer":         # the offset-producing convolution has dilation 1 and the operator's size rule
            case["offset_std"] = round(rng.uniform(0.2, 1.0), 2)
        t = _counts(case)
        if _contraction(case) <= kind["flops"] and t["corners"] <= kind["corners"] and 4 * (t["x"] + t["y"] + t["off"]) < 2e9:
            return case
