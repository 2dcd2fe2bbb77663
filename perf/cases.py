"""Performance cases: the work users of this package have it do, through its public entry points.

A case is a dict of plain values; its "kind" says which entry points a pass goes through:

    linear     ops.quant_rows + ops.gemm_plain: one quantised Linear (16-bit or fp32 rows in, bf16 out)
    attention  ops.attn_fwd on a [3, B, N, H, 64] tensor
    swap       linear_swap.enable: the four swapped Linears of a block, called the way the torch model calls them
    model      stack.make_variant: one model_fn call on normalised images, eager or as a captured CUDA graph
    frames     device-resident uint8 frames -> ops.resize_norm -> model_fn -> ops.semantic, as a captured CUDA graph
    video      host frames through pipeline.VideoPipeline.run, labels back on the host

listed() is one case per use; draw() gives further cases of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lightly_trian_quant_b200 import linear_swap, modeldef, ops, pipeline, stack

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
ARCHS = {"vit_b": modeldef.VIT_B, "vit_l": modeldef.VIT_L}
BITS = {"mx8": 8 + 8 / 32, "nv4": 4 + 8 / 16, "mx4": 4 + 8 / 32, "bf16": 16.0}      # bits per stored value, scales included


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one fc1 of a single 640 x 640 frame (1600 patches + cls + 4 registers): the smallest call, launch latency counts
        dict(name="linear_mx8_1_frame", kind="linear", fmt="mx8", rows=1605, k=1024, n=4096, dtype="bf16"),
        # fc2 of 32 frames: the largest single Linear of the quantise + GEMM sweep
        dict(name="linear_nv4_32_frames", kind="linear", fmt="nv4", rows=1605 * 32, k=4096, n=1024, dtype="bf16"),
        # one frame's attention with the queries joined, 1805 tokens: odd, ends inside a tile
        dict(name="attention_f16_1_frame", kind="attention", dtype="f16", batch=1, tokens=1805, heads=12),
        # a torch model with the Linears of a block swapped; NVFP4 measures its activation scale on every call
        dict(name="swap_vit_b_nv4_4_frames", kind="swap", arch="vit_b", fmt="nv4", rows=1605 * 4),
        # a thumbnail through the whole small model, called eagerly: host time and launches
        dict(name="model_vit_b_mx8_256px_1", kind="model", arch="vit_b", fmt="mx8", flags="", size=256, batch=1, graph=False),
        # live video, one frame at a time: the latency of a frame
        dict(name="model_vit_l_nv4_640px_1", kind="model", arch="vit_l", fmt="nv4", flags="", size=640, batch=1, graph=True),
        # the throughput step of the benchmark: 14 frames of 1900 x 1440 to labels and scores
        dict(name="frames_vit_l_nv4_640px_14", kind="frames", arch="vit_l", fmt="nv4", flags="", size=640, batch=14, height=1440, width=1900),
        # the ViT-B configuration on images that are already normalised
        dict(name="model_vit_b_mx8_640px_14", kind="model", arch="vit_b", fmt="mx8", flags="", size=640, batch=14, graph=True),
        # the high-resolution configuration: 4096 patches, attention in f16; the largest step
        dict(name="model_vit_l_mx4_f16_1024px_8", kind="model", arch="vit_l", fmt="mx4", flags="+f16attn", size=1024, batch=8, graph=True),
        # unquantised linears, a few images, eager
        dict(name="model_vit_b_bf16_640px_3", kind="model", arch="vit_b", fmt="bf16", flags="", size=640, batch=3, graph=False),
        # three micro-batches of host frames, one numpy array per frame as a decoder gives them
        dict(name="video_vit_l_nv4_42", kind="video", arch="vit_l", fmt="nv4", flags="", size=640, batch=14, frames=42, height=1440, width=1900),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "attention", "swap", "model", "model", "model", "frames", "video"])
    fmt = rng.choice(["mx8", "nv4", "mx4"])
    arch = rng.choice(["vit_b", "vit_l"])
    if kind == "linear":
        d = ARCHS[arch].dim
        k, n = rng.choice([(d, 3 * d), (d, d), (d, 4 * d), (4 * d, d), (rng.randrange(1, 17) * 256, rng.randrange(1, 33) * 128)])
        return dict(kind=kind, fmt=fmt, rows=_log(rng, 1, 51360), k=k, n=n, dtype=rng.choice(["bf16", "bf16", "f16", "f32"]))
    if kind == "attention":
        return dict(kind=kind, dtype=rng.choice(["bf16", "f16"]), batch=_log(rng, 1, 14), tokens=_log(rng, 64, 4301), heads=rng.choice([12, 16]))
    if kind == "swap":
        return dict(kind=kind, arch=arch, fmt=fmt, rows=_log(rng, 197, 1605 * 8))
    flags = rng.choice(["", "", "+f16attn", "+fp32pts", "+bf16head"])
    size = 64 * rng.choice([2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16])
    most = min(16, 8 * 1024 * 1024 // (size * size), int(40e9 / (size // 16) ** 4) + 1)
    batch = _log(rng, 1, max(1, most))
    if kind == "model":
        if rng.random() < 0.15:
            fmt, flags = "bf16", ""
        return dict(kind=kind, arch=arch, fmt=fmt, flags=flags, size=size, batch=batch, graph=rng.random() < 0.6)
    size, batch = min(size, 640), min(batch, 14)
    height, width = _log(rng, 360, 1440), _log(rng, 480, 1920)
    case = dict(kind=kind, arch=arch, fmt=fmt, flags=flags, size=size, batch=batch, height=height, width=width)
    if kind == "video":
        case["frames"] = rng.randrange(batch, 3 * batch + 1)
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(gen, rows, k, dtype):
    """N(0, 1) with one channel in a hundred 20 times larger, the outliers that block scales exist for."""
    x = torch.randn(rows, k, generator=gen, device="cuda")
    x[:, torch.randperm(k, generator=gen, device="cuda")[: max(1, k // 100)]] *= 20
    return x.to(dtype)


@torch.no_grad()
def _model(cfg, gen):
    """The torch model with the upstream initialisation (normal 0.02 linears, LayerScale 1e-5), made on the GPU."""
    with torch.device("cuda"):
        model = modeldef.DINOv3EoMTSemanticSegmentation(cfg)
    for m in model.modules():
        if isinstance(m, torch.nn.Linear):
            m.weight.normal_(0.0, 0.02, generator=gen)
            m.bias.zero_()
        elif isinstance(m, torch.nn.LayerNorm):
            m.weight.fill_(1.0)
            m.bias.zero_()
        elif isinstance(m, (torch.nn.Conv2d, torch.nn.ConvTranspose2d)):
            bound = (m.weight[0].numel() if isinstance(m, torch.nn.Conv2d) else 4 * m.weight.shape[0]) ** -0.5
            m.weight.uniform_(-bound, bound, generator=gen)
            if m.bias is not None:
                m.bias.uniform_(-bound, bound, generator=gen)
    model.backbone.cls_token.normal_(0.0, 0.02, generator=gen)
    model.backbone.storage_tokens.normal_(0.0, 0.02, generator=gen)
    model.queries.weight.normal_(0.0, 1.0, generator=gen)
    return model.eval()


def _variant(case, gen):
    name = f"b200_{case['fmt']}{case['flags']}+s{case['size']}"
    return stack.make_variant(case["arch"], _model(ARCHS[case["arch"]], gen), name)


def _frames(gen, count, height, width):
    """Smooth content (an upsampled 6 x 8 grid) plus camera noise of sigma 8, uint8 [count, height, width, 3] on the GPU."""
    out = torch.empty(count, height, width, 3, dtype=torch.uint8, device="cuda")
    for i in range(count):
        low = torch.rand(1, 3, 6, 8, generator=gen, device="cuda") * 255.0
        img = torch.nn.functional.interpolate(low, size=(height, width), mode="bilinear", align_corners=False)[0]
        img += torch.randn(3, height, width, generator=gen, device="cuda") * 8.0
        out[i] = img.clamp(0, 255).permute(1, 2, 0).to(torch.uint8)
    return out


def _captured(fn):
    """fn as a user captures it: the first call eagerly (static scales are measured), then one CUDA graph."""
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    return graph, out


@torch.no_grad()
def prepare(case, seed):
    torch.set_grad_enabled(False)
    gen = _gen(seed)
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "linear":
        rows, k, n, fmt = case["rows"], case["k"], case["n"], case["fmt"]
        state["x"] = _activations(gen, rows, k, DTYPES[case["dtype"]])
        state["w"] = ops.QWeight(torch.randn(n, k, generator=gen, device="cuda") * 0.02, fmt)
        state["bias"] = (torch.randn(n, generator=gen, device="cuda") * 0.02).to(torch.bfloat16).float()
        state["buf"] = ops.ActBuf(rows, k, fmt)
        if fmt == "nv4":
            stack.set_ts(state["buf"].ts, state["x"])
    elif kind == "attention":
        state["qkv"] = torch.randn(3, case["batch"], case["tokens"], case["heads"], 64, generator=gen, device="cuda").to(DTYPES[case["dtype"]])
    elif kind == "swap":
        cfg = ARCHS[case["arch"]]
        one = modeldef.EoMTConfig(dim=cfg.dim, depth=1, heads=cfg.heads, ffn=cfg.ffn)
        model = _model(one, gen).to(torch.bfloat16)
        linear_swap.enable(model, [(0, unit) for unit in ("qkv", "proj", "fc1", "fc2")], fmt=case["fmt"])
        state["model"] = model
        state["x"] = torch.randn(1, case["rows"], cfg.dim, generator=gen, device="cuda").to(torch.bfloat16)
        state["o"] = torch.randn(1, case["rows"], cfg.dim, generator=gen, device="cuda").to(torch.bfloat16) * 0.2
    elif kind == "model":
        fn, _ = _variant(case, gen)
        x = torch.rand(case["batch"], 3, case["size"], case["size"], generator=gen, device="cuda")
        mean, std = (torch.tensor(v, device="cuda").view(1, 3, 1, 1) for v in (ops.IMAGENET_MEAN, ops.IMAGENET_STD))
        x = ((x - mean) / std).to(torch.bfloat16).contiguous()
        state["fn"], state["x"] = fn, x
        if case["graph"]:
            state["graph"], state["out"] = _captured(lambda: fn(x))
        else:
            fn(x)
    elif kind == "frames":
        fn, _ = _variant(case, gen)
        frames = _frames(gen, case["batch"], case["height"], case["width"])

        def whole():
            masks, classes = fn(ops.resize_norm(frames, case["size"]))
            labels, scores = ops.semantic(masks, classes, want_scores=True)
            return {"masks": masks, "classes": classes, "labels": labels, "scores": scores}

        state["fn"], state["x"] = fn, frames
        state["graph"], state["out"] = _captured(whole)
    else:
        fn, pipe_cls = _variant(case, gen)
        frames = _frames(gen, case["frames"], case["height"], case["width"])
        video = pipeline.VideoPipeline(pipe_cls(None, fn, case["size"]), case["batch"], case["height"], case["width"])
        video.warmup(frames[: case["batch"]])
        state["video"] = video
        state["frames"] = list(frames.cpu().numpy())
        state["side"] = case["size"] // 4
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return ops.gemm_plain(ops.quant_rows(state["x"], state["buf"]), state["w"], state["bias"])
    if kind == "attention":
        return ops.attn_fwd(state["qkv"])
    if kind == "swap":
        block, x = state["model"].backbone.blocks[0], state["x"]
        return [block.attn.qkv(block.norm1(x)), block.attn.proj(state["o"]), block.mlp(block.norm2(x))]
    if kind == "video":
        labels = np.empty((len(state["frames"]), state["side"], state["side"]), dtype=np.uint8)

        def keep(index, picture):
            labels[index] = picture

        state["video"].run(state["frames"], keep)
        return labels
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return state["fn"](state["x"])


# ------------------------------------------------------------------------------------------------ floors and tolerances
def _model_work(case, batch):
    """flops of a model_fn call; bytes of its weights, its images and its two outputs."""
    cfg = ARCHS[case["arch"]]
    d, ff, Q = cfg.dim, cfg.ffn, cfg.num_queries
    P = (case["size"] // 16) ** 2
    flops = 2.0 * batch * P * 768 * d                                                        # patch embedding
    for i in range(cfg.depth):
        tokens = P + 1 + cfg.n_storage_tokens + (Q if i >= cfg.depth - cfg.num_joint_blocks else 0)
        flops += 2.0 * batch * tokens * (4 * d * d + 2 * d * ff) + 4.0 * batch * tokens * tokens * d
    flops += 2.0 * batch * (P + 4 * P) * d * 4 * d + 18.0 * batch * (4 * P + 16 * P) * d        # the two up-scaling stages
    flops += 2.0 * batch * Q * d * (3 * d + cfg.num_classes + 1) + 2.0 * batch * Q * d * 16 * P   # mask MLP, classes, mask product
    head = "bf16" if "bf16head" in case["flags"] else case["fmt"]
    weights = cfg.depth * (4 * d * d + 2 * d * ff) * BITS[case["fmt"]] / 8 + 2 * 4 * d * d * BITS[head] / 8 + (768 * d + 3 * d * d) * 2
    return flops, weights, batch * 3 * case["size"] ** 2 * 2, batch * Q * (16 * P + cfg.num_classes + 1) * 2


def work(case):
    kind = case["kind"]
    if kind == "linear":
        rows, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": rows * k * (4 if case["dtype"] == "f32" else 2) + n * k * BITS[case["fmt"]] / 8 + n * 4 + rows * n * 2, "flops": 2.0 * rows * k * n}
    if kind == "attention":
        b, t, h = case["batch"], case["tokens"], case["heads"]
        return {"bytes": 4 * b * t * h * 64 * 2, "flops": 4.0 * b * h * t * t * 64}
    if kind == "swap":
        cfg, rows = ARCHS[case["arch"]], case["rows"]
        values = 4 * cfg.dim ** 2 + 2 * cfg.dim * cfg.ffn
        return {"bytes": values * BITS[case["fmt"]] / 8 + rows * cfg.dim * 2 * (2 + 5), "flops": 2.0 * rows * values}
    if kind == "model":
        flops, weights, images, outputs = _model_work(case, case["batch"])
        return {"bytes": weights + images + outputs, "flops": flops}
    pixels = case["height"] * case["width"] * 3
    if kind == "frames":
        flops, weights, _, outputs = _model_work(case, case["batch"])
        labels = case["batch"] * (case["size"] // 4) ** 2
        return {"bytes": weights + case["batch"] * pixels + outputs + labels * (1 + 4 * 3), "flops": flops}
    flops, weights, _, _ = _model_work(case, case["frames"])
    return {"bytes": weights + case["frames"] * (pixels + (case["size"] // 4) ** 2), "flops": flops}


def tolerance(case):
    """Relative errors of another correct implementation at the same precision."""
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 2e-3, "max": 1e-2}                       # the same codes, fp32 sums in another order, one rounding to bf16
    if kind == "attention":
        return {"rel": 1e-3, "max": 2e-2} if case["dtype"] == "f16" else {"rel": 4e-3, "max": 5e-2}      # P and O rounded to 16 bits
    if kind == "swap":
        return {"rel": 1e-2, "max": 0.2}                        # a hidden value at a rounding boundary moves its code by a whole step
    if kind == "video":
        return {"differ": 1e-2}                                 # pixels whose two best classes are within rounding of each other
    return {"rel": 1e-2, "max": 0.2, "differ": 1e-2}            # bf16 rounding points and codes at rounding boundaries
