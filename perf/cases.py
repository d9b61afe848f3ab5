"""Performance cases of the ConvNN-Attention forward path, through the package's public entry points.

``listed()`` are fixed cases, ``draw(rng)`` gives further ones of the same ranges.  Two kinds:

  vit    the whole model, ``convnn_b200.ViT`` (bfloat16 or float32, float or 8-bit images), called on a
         batch as an inference program calls it, or with ``lanes`` > 1 through ``ForwardLanes``, the
         throughput runner with that many batches in flight;
  layer  the standalone ``MultiHeadConvNNAttention`` module on (B, T, D) tokens.

``prepare`` makes what such a program holds before the call (model with seeded random weights, inputs on the
GPU, for ``lanes`` the captured graphs), ``run`` is one pass.
"""
from __future__ import annotations

import math

import torch

import convnn_b200

# d_hidden, d_mlp, heads of the 197-token models
SIZES = {"tiny": (192, 768, 3), "small": (384, 1536, 6), "base": (768, 3072, 12)}
LAYERS = 12


def _vit(name, size, layer, batch, img=224, patch=16, heads=1, dtype="bf16", images="float", metric="cosine",
         sampling="all", samples=-1, conv="depthwise", K=9, coord=False, classes=1000, lanes=1):
    c = dict(kind="vit", size=size, layer=layer, batch=batch, img=img, patch=patch, heads=heads, dtype=dtype,
             images=images, metric=metric, sampling=sampling, samples=samples, conv=conv, K=K, coord=coord,
             classes=classes, lanes=lanes)
    if name:
        c["name"] = name
    return c


def _layer(name, batch, tokens, d, heads=1, dtype="bf16", metric="cosine", sampling="all", samples=-1,
           conv="depthwise", K=9, coord=False):
    c = dict(kind="layer", batch=batch, tokens=tokens, d=d, heads=heads, dtype=dtype, metric=metric,
             sampling=sampling, samples=samples, conv=conv, K=K, coord=coord)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one image, the latency of an interactive request
        _vit("vit_tiny_bf16_b1", "tiny", "ConvNNAttention", 1),
        # a ragged serving batch of decoded 8-bit images, normalised on the way in
        _vit("vit_tiny_bf16_u8_b37", "tiny", "ConvNNAttention", 37, images="uint8"),
        # an evaluation loop's batch, ViT-Tiny at 224 x 224: the workload of bench.py, one batch at a time
        _vit("vit_tiny_bf16_b256", "tiny", "ConvNNAttention", 256),
        # the same model served for throughput, two batches in flight
        _vit("vit_tiny_bf16_lanes2_b256", "tiny", "ConvNNAttention", 256, lanes=2),
        # float32 on CIFAR-sized images: the configuration whose results are compared with the CPU's
        _vit("vit_tiny_fp32_32px_b32", "tiny", "ConvNNAttention", 32, img=32, patch=4, dtype="fp32", classes=10),
        # ViT-Small, euclidean distance to 64 random candidates, depthwise-separable conv
        _vit("vit_small_rand64_sep_b256", "small", "ConvNNAttention", 256, metric="euclidean", sampling="random",
             samples=64, conv="depthwise-separable"),
        # ViT-Base, half softmax attention and half ConvNN (standard conv), 12 heads
        _vit("vit_base_branchattn_b128", "base", "BranchAttention", 128, heads=12, conv="standard"),
        # the command line's default heads and similarity with the Conv1d branch
        _vit("vit_tiny_branchconv_b64", "tiny", "BranchConv", 64, heads=3, metric="matmul"),
        # float32 layer, several heads, strided candidates, standard conv
        _layer("layer_fp32_h3_spatial_std", 8, 197, 192, heads=3, dtype="fp32", metric="matmul", sampling="spatial",
               samples=49, conv="standard"),
        # 577 tokens (384 x 384 at patch 16) with the coordinate channel, ragged batch and candidate count
        _layer("layer_coord_rand_sep", 7, 577, 384, metric="euclidean", sampling="random", samples=150,
               conv="depthwise-separable", coord=True, K=16),
        # long sequences: 64 x 64 patches against every token ...
        _layer("layer_n4096_all_k9", 8, 4096, 768),
        # ... and 128 x 128 patches against a strided grid, long neighbour lists
        _layer("layer_n16384_spatial_k25", 8, 16384, 768, sampling="spatial", samples=4096, K=25),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _options(rng, dtype):
    conv = rng.choice(["depthwise", "depthwise", "standard", "depthwise-separable"])
    coord = conv != "depthwise" and rng.random() < 0.25
    return dict(metric=rng.choice(["cosine", "cosine", "matmul", "euclidean"]), conv=conv, coord=coord, dtype=dtype,
                K=rng.choice([5, 9, 9, 9, 16, 25]))


def _draw(rng):
    dtype = "bf16" if rng.random() < 0.75 else "fp32"
    opts = _options(rng, dtype)
    sampling = rng.choice(["all", "all", "random", "spatial"])
    if rng.random() < 0.55:
        size = rng.choice(["tiny", "tiny", "small", "base"])
        layer = rng.choice(["ConvNNAttention", "ConvNNAttention", "ConvNNAttention", "BranchAttention", "BranchConv"])
        img, patch, classes = rng.choice([(224, 16, 1000), (224, 16, 1000), (32, 4, 10), (64, 8, 100)])
        tokens = (img // patch) ** 2 + 1
        # several heads need the module's default sequence length of 197 tokens
        heads = SIZES[size][2] if tokens == 197 and rng.random() < 0.5 else 1
        samples = -1 if sampling == "all" else rng.randint(max(32, opts["K"]), tokens)
        lanes = 2 if dtype == "bf16" and rng.random() < 0.2 else 1
        images = "uint8" if rng.random() < 0.25 else "float"
        return _vit(None, size, layer, _log_int(rng, 1, 256), img=img, patch=patch, heads=heads, images=images,
                    sampling=sampling, samples=samples, classes=classes, lanes=lanes, **opts)
    tokens = _log_int(rng, 50, 16384)
    d = rng.choice([192, 256, 384, 512, 768])
    heads = rng.choice([1, 1, 2, 4]) if tokens < 2048 else 1
    samples = -1 if sampling == "all" else _log_int(rng, max(32, opts["K"]), max(33, tokens // 2))
    return _layer(None, _log_int(rng, 1, max(1, min(256, 131072 // tokens))), tokens, d, heads=heads,
                  sampling=sampling, samples=samples, **opts)


def _cost(case):
    """Size of a case in bfloat16 operations: float32 and the coordinate channel cannot use 16-bit products, and
    their K * d_k wide standard conv weighs most."""
    flops = work(case)["flops"]
    if case["dtype"] == "fp32" or case["coord"]:
        flops *= 64
        if case["conv"] == "standard":
            d = case["d"] if case["kind"] == "layer" else SIZES[case["size"]][0]
            flops *= 4 if d // case["heads"] <= 384 else 16
    return flops


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        rows = case["batch"] * (_tokens(case))
        d = case["d"] if case["kind"] == "layer" else SIZES[case["size"]][0]
        if _cost(case) <= most and rows * case["K"] * (d + 8 * case["heads"]) < 1 << 30:
            return case


def _tokens(case):
    return case["tokens"] if case["kind"] == "layer" else (case["img"] // case["patch"]) ** 2 + 1


def _vary_taps(module, gen):
    """The modules start depthwise taps at 1; trained taps differ from each other."""
    for m in module.modules():
        if isinstance(m, torch.nn.Conv1d) and m.groups > 1:
            m.weight.add_(torch.randn(m.weight.shape, device="cuda", generator=gen), alpha=0.25)


def _vit_parts(case):
    d, d_mlp, _ = SIZES[case["size"]]
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    args = convnn_b200.make_args(
        layer=case["layer"], img_size=(3, case["img"], case["img"]), patch_size=case["patch"], num_layers=LAYERS,
        num_heads=case["heads"], d_hidden=d, d_mlp=d_mlp, num_classes=case["classes"], K=case["K"],
        magnitude_type=case["metric"], sampling_type=case["sampling"], num_samples=case["samples"],
        convolution_type=case["conv"], coordinate_encoding=case["coord"], dropout=0.0, attention_dropout=0.0)
    with torch.device("cuda"):
        model = convnn_b200.ViT(args)
    return model.to(dtype).eval(), dtype


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        if case["kind"] == "layer":
            dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
            with torch.device("cuda"):
                model = convnn_b200.MultiHeadConvNNAttention(
                    case["d"], case["heads"], 0.0, case["K"], case["sampling"], case["samples"], 0, case["metric"],
                    seq_length=case["tokens"], coordinate_encoding=case["coord"], convolution_type=case["conv"])
            model = model.to(dtype).eval()
            _vary_taps(model, gen)
            if case["sampling"] == "random":      # one candidate set, so that passes can be compared
                model.candidate_override = torch.randperm(case["tokens"], generator=gen, device="cuda")[: case["samples"]]
            x = torch.randn(case["batch"], case["tokens"], case["d"], device="cuda", generator=gen).to(dtype)
            return {"model": model, "x": x}
        model, dtype = _vit_parts(case)
        _vary_taps(model, gen)
        if case["sampling"] == "random":
            model.set_candidates(torch.randperm(_tokens(case), generator=gen, device="cuda")[: case["samples"]])
        shape = (case["batch"], 3, case["img"], case["img"])
        xs = [torch.randint(0, 256, shape, device="cuda", generator=gen, dtype=torch.uint8) if case["images"] == "uint8"
              else torch.randn(shape, device="cuda", generator=gen).to(dtype) for _ in range(case["lanes"])]
        if case["lanes"] > 1:
            # the captured graphs read the weights and the inputs where they lie: the program keeps both
            return {"lanes": convnn_b200.ForwardLanes(model, xs, lanes=case["lanes"]), "model": model, "xs": xs}
        return {"model": model, "x": xs[0]}


def run(state):
    with torch.no_grad():
        if "lanes" in state:
            return state["lanes"].replay(0)
        return state["model"](state["x"])


def _convnn_work(case, rows, T, d):
    """(flops, weight values) of one ConvNN layer of width d over ``rows`` tokens in sequences of T."""
    S = T if case["sampling"] == "all" else case["samples"]
    q_rows = rows // T * S
    dk = d // case["heads"]
    C = dk + (1 if case["coord"] else 0)
    n_heads = case["heads"]
    flops = 2.0 * (2 * rows + q_rows) * d * d + 2.0 * rows * S * n_heads * C + 2.0 * rows * d * d
    weights = 4 * d * d
    if case["conv"] == "standard":
        flops += 2.0 * rows * n_heads * case["K"] * C * dk
        weights += case["K"] * C * dk
    else:
        flops += 2.0 * rows * n_heads * case["K"] * C
        weights += case["K"] * C
        if case["conv"] == "depthwise-separable":
            flops += 2.0 * rows * n_heads * C * dk
            weights += C * dk
    return flops, weights


def work(case):
    """One pass: the operations of the layers' definitions; inputs and weights read once, outputs written once."""
    elt = 2 if case["dtype"] == "bf16" else 4
    T = _tokens(case)
    rows = case["batch"] * T
    if case["kind"] == "layer":
        flops, weights = _convnn_work(case, rows, T, case["d"])
        return {"bytes": float(elt * (2 * rows * case["d"] + weights)), "flops": flops}
    d, d_mlp, _ = SIZES[case["size"]]
    half = d // 2
    if case["layer"] == "ConvNNAttention":
        flops, weights = _convnn_work(case, rows, T, d)
    else:
        flops, weights = _convnn_work(case, rows, T, half)
        if case["layer"] == "BranchAttention":
            flops += 2.0 * rows * 4 * half * half + 4.0 * rows * T * half
            weights += 4 * half * half
        else:
            taps = 9 * (half // case["heads"])
            flops += 2.0 * rows * (2 * half * half + half * taps)
            weights += 2 * half * half + taps * (half // case["heads"])
        flops += 2.0 * rows * d * d
        weights += d * d
    flops += 4.0 * rows * d * d_mlp
    weights += 2 * d * d_mlp
    pixels = 3 * case["patch"] ** 2
    flops = LAYERS * flops + 2.0 * (rows - case["batch"]) * d * pixels + 2.0 * case["batch"] * d * case["classes"]
    weights = LAYERS * weights + d * (pixels + T + case["classes"])
    image_bytes = case["batch"] * 3 * case["img"] ** 2 * (1 if case["images"] == "uint8" else elt)
    n = case["lanes"]
    return {"bytes": float(n * (image_bytes + elt * case["batch"] * case["classes"]) + elt * weights), "flops": n * flops}


def tolerance(case):
    # A layer's result is a continuous function of its inputs except where two candidates are within rounding of
    # each other: there another neighbour order is as right, and a few rows differ by the size of their values
    # ("max").  bfloat16 rounds q, k, v, the conv's result and the output once each; a model does so twelve times.
    if case["dtype"] == "fp32":
        return {"rel": 1e-4, "max": 0.9}
    return {"rel": 1e-2 if case["kind"] == "layer" else 2e-2, "max": 0.9}
