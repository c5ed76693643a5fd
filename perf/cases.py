"""What a user of this package has it do, as cases that can be timed.

Three public entry points, each in inference and in training (forward + backward):

* ``op``       ``registry.msda`` on locations and normalised weights: what the attention cores of
               Deformable-DETR style models call.
* ``offsets``  ``registry.msda_from_offsets`` on reference points, predicted offsets and raw
               logits: what a layer of one's own calls.
* ``layer``    ``nn.MultiScaleDeformAttn2d`` with its four projections.

``queries = 0`` is the encoder: every pixel of the pyramid is a query, its reference point the
pixel's centre.  ``queries > 0`` is a decoder: that many queries with reference points anywhere
in the image.  Values, logits and upstream gradients are N(0, 1), samples lie N(0, 0.05) of the
image around their reference point (a few percent outside it), weights are softmax-normalised
unless the call normalises them itself.
"""

from __future__ import annotations

import math

import torch

from deformops_b200.nn import MultiScaleDeformAttn2d
from deformops_b200.registry import msda, msda_from_offsets

_DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}

# Pyramids of the package's own configurations: pixel decoders at 512 and 1024 pixels, the
# detection encoder's 800 x 1066 image, and the small one its CPU configuration uses.
_PYRAMID_512 = "64x64,32x32,16x16"
_PYRAMID_1024 = "128x128,64x64,32x32"
_PYRAMID_DETR = "100x134,50x67,25x34,13x17"
_PYRAMID_SMALL = "32x32,16x16,8x8"


def _case(name, entry, train, dtype, batch, levels, queries=0, heads=8, head_dim=32, points=4,
          boxes=False):
    return {"name": name, "entry": entry, "train": train, "dtype": dtype, "batch": batch,
            "levels": levels, "queries": queries, "heads": heads, "head_dim": head_dim,
            "points": points, "boxes": boxes}


def listed():
    return [
        # one image through a decoder layer at serving time: the smallest call, all latency
        _case("decoder_infer_f16", "op", False, "float16", 1, _PYRAMID_DETR, queries=300),
        # a decoder layer in training: few queries, but a whole grad_value to produce
        _case("decoder_train_f16", "op", True, "float16", 4, _PYRAMID_DETR, queries=300),
        # the same layer with box reference points, softmax and offsets left to the call
        _case("decoder_boxes_train_bf16", "offsets", True, "bfloat16", 2, _PYRAMID_DETR,
              queries=900, boxes=True),
        # small float32 encoder: fine-tuning and tests at full precision
        _case("encoder_small_train_f32", "op", True, "float32", 2, _PYRAMID_SMALL),
        # one 1024-pixel image through an encoder layer at serving time
        _case("encoder_1024_infer_bf16", "op", False, "bfloat16", 1, _PYRAMID_1024),
        # pixel-decoder training at 512 pixels, an ordinary batch
        _case("encoder_512_train_bf16", "op", True, "bfloat16", 8, _PYRAMID_512),
        # pixel-decoder training at 1024 pixels, the headline shape
        _case("encoder_1024_train_bf16", "op", True, "bfloat16", 4, _PYRAMID_1024),
        # detection encoder training: four levels of odd sizes, float16 and float32
        _case("encoder_detr_train_f16", "op", True, "float16", 4, _PYRAMID_DETR),
        _case("encoder_detr_train_f32", "op", True, "float32", 4, _PYRAMID_DETR),
        # a ragged pyramid with other head and point counts, softmax inside the call
        _case("encoder_ragged_train_bf16", "offsets", True, "bfloat16", 3, "75x113,38x57,19x29",
              heads=6, head_dim=64, points=3),
        # the whole layer with its projections, an encoder layer of pixel-decoder training
        _case("layer_512_train_bf16", "layer", True, "bfloat16", 8, _PYRAMID_512),
        # a large batch of the headline shape: one device's share of a global batch of 64
        _case("encoder_1024_batch16_train_bf16", "op", True, "bfloat16", 16, _PYRAMID_1024),
    ]


def _levels(case):
    return [tuple(int(x) for x in level.split("x")) for level in case["levels"].split(",")]


def _dims(case):
    levels = _levels(case)
    S = sum(h * w for h, w in levels)
    return case["batch"], S, case["queries"] or S, len(levels)


def _cost(case):
    B, S, Q, L = _dims(case)
    channels = case["heads"] * case["head_dim"]
    passes = 3 if case["train"] else 1
    width = 2 if case["dtype"] == "float32" else 1
    return passes * width * B * channels * (Q * L * case["points"] + S)


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        # image of any aspect ratio, finest level at a quarter or an eighth of its side
        height = _log_uniform(rng, 24, 160)
        width = max(24, min(200, int(height * rng.uniform(0.7, 1.5))))
        levels = []
        for _ in range(rng.choice([3, 3, 4, 4, 5])):
            levels.append(f"{height}x{width}")
            height, width = (height + 1) // 2, (width + 1) // 2
        heads, head_dim = rng.choice([(8, 32), (8, 32), (8, 32), (8, 16), (6, 64), (4, 64), (16, 32)])
        entry = rng.choice(["op", "op", "op", "offsets", "offsets", "layer"])
        queries = 0 if rng.random() < 0.6 else _log_uniform(rng, 50, 1800)
        points = rng.choice([4, 4, 4, 8] if len(levels) == 5 else [4, 4, 4, 3, 8])
        case = _case("", entry, rng.random() < 0.7,
                     rng.choice(["bfloat16", "bfloat16", "float16", "float32"]),
                     _log_uniform(rng, 1, 16), ",".join(levels), queries, heads, head_dim,
                     points, queries > 0 and entry != "op" and rng.random() < 0.5)
        del case["name"]
        if _cost(case) <= most:
            return case


def _reference_points(case, gen):
    """(B, Q, 1, 2) centres as (x, y)."""
    B, _, Q, _ = _dims(case)
    if case["queries"]:
        return torch.rand(B, Q, 1, 2, generator=gen, device="cuda")
    rows = []
    for h, w in _levels(case):
        y, x = torch.meshgrid((torch.arange(h, device="cuda") + 0.5) / h,
                              (torch.arange(w, device="cuda") + 0.5) / w, indexing="ij")
        rows.append(torch.stack([x.reshape(-1), y.reshape(-1)], -1))
    return torch.cat(rows).view(1, Q, 1, 2).expand(B, Q, 1, 2)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    dtype = _DTYPES[case["dtype"]]
    B, S, Q, L = _dims(case)
    G, D, K = case["heads"], case["head_dim"], case["points"]

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    shapes = torch.tensor(_levels(case), dtype=torch.int64, device="cuda")
    sizes = shapes[:, 0] * shapes[:, 1]
    state = {"entry": case["entry"], "train": case["train"], "shapes": shapes,
             "starts": torch.cumsum(sizes, 0) - sizes}
    centres = _reference_points(case, gen)
    spread = 0.05 * normal(B, Q, G, L, K, 2)
    if case["boxes"]:
        # boxes of a tenth to half the image; an offset of K moves a sample by half a box
        box = 0.1 + 0.4 * torch.rand(B, Q, 1, 2, generator=gen, device="cuda")
        reference = torch.cat([centres, box], -1).expand(B, Q, L, 4).contiguous()
        offsets = spread * (2 * K) / box.view(B, Q, 1, 1, 1, 2)
    else:
        reference = centres.expand(B, Q, L, 2).contiguous()
        offsets = spread * shapes.flip(-1).view(1, 1, 1, L, 1, 2)          # pixels of each level
    if case["entry"] == "layer":
        torch.manual_seed(int(seed))
        layer = MultiScaleDeformAttn2d(G * D, num_heads=G, num_levels=L, num_points=K)
        with torch.no_grad():
            # trained layers predict offsets and weights from the query, not from the bias alone
            layer.proj_offset.weight.normal_(0.0, 2.0 / math.sqrt(G * D))
            layer.proj_weights.weight.normal_(0.0, 1.0 / math.sqrt(G * D))
        state["layer"] = layer.to("cuda", dtype)
        inputs = [normal(B, Q, G * D).to(dtype), normal(B, S, G * D).to(dtype)]
        state["reference"] = reference
    elif case["entry"] == "offsets":
        inputs = [normal(B, S, G, D).to(dtype), offsets.to(dtype), normal(B, Q, G, L * K).to(dtype)]
        state["reference"] = reference
    else:
        weights = torch.softmax(normal(B, Q, G, L * K), -1).to(dtype)
        inputs = [normal(B, S, G, D).to(dtype), centres.view(B, Q, 1, 1, 1, 2) + spread, weights]
    state["inputs"] = [t.requires_grad_(case["train"]) for t in inputs]
    if case["train"]:
        state["grad"] = normal(B, Q, G * D).to(dtype)
    return state


def _forward(state):
    shapes, starts, inputs = state["shapes"], state["starts"], state["inputs"]
    if state["entry"] == "op":
        value, locations, weights = inputs
        return msda(value, shapes, starts, locations, weights)
    if state["entry"] == "offsets":
        value, offsets, logits = inputs
        return msda_from_offsets(value, shapes, starts, state["reference"], offsets, logits,
                                 method="softmax")
    query, memory = inputs
    return state["layer"](query, state["reference"], memory, shapes, starts)


def run(state):
    if not state["train"]:
        with torch.no_grad():
            return [_forward(state)]
    out = _forward(state)
    wanted = list(state["inputs"])
    if state["entry"] == "layer":
        wanted += list(state["layer"].parameters())
    return [out.detach(), *torch.autograd.grad(out, wanted, state["grad"])]


def work(case):
    """Each operand read once, each result written once; four corners per point and channel
    (multiply-add each), three times that backward, plus the layer's matrix products."""
    B, S, Q, L = _dims(case)
    G, D, K = case["heads"], case["head_dim"], case["points"]
    e = 4 if case["dtype"] == "float32" else 2
    C, P = G * D, L * K
    value, rows, points = B * S * C * e, B * Q * C * e, B * Q * G * P
    flops = 8 * points * D
    if case["entry"] == "layer":
        tokens = value + rows + B * Q * L * (16 if case["boxes"] else 8)     # memory, query, reference
        weights = (2 * C * C + 3 * G * P * C) * e
        products = 2 * B * (S * C * C + Q * C * C + Q * C * 3 * G * P)
        forward = tokens + weights + rows
        backward = tokens + weights + rows + value + rows + weights
        flops += products
        return {"bytes": forward + (backward if case["train"] else 0),
                "flops": 3 * flops if case["train"] else flops}
    if case["entry"] == "offsets":
        spots, reference = points * 2 * e, B * Q * L * (16 if case["boxes"] else 8)
    else:
        spots, reference = points * 2 * 4, 0
    inputs = value + spots + points * e
    forward = inputs + reference + rows
    backward = inputs + reference + rows + inputs
    return {"bytes": forward + (backward if case["train"] else 0),
            "flops": 3 * flops if case["train"] else flops}


def tolerance(case):
    # 16-bit results carry the type's own rounding; float32 sums of many terms, in any order
    if case["dtype"] == "float32":
        # the layer's float32 locations pass through matrix products of either order
        return {"rel": 1e-4 if case["entry"] == "layer" else 1e-5, "max": 1e-3}
    return {"rel": 1e-2, "max": 0.25}
