"""What a user of this package has it do, as measurable cases: the operators called one by one the way a patched model
calls them, a scene of attention layers launched from Python or replayed from a CUDA graph, and the accelerated blocks.

Every case is a dict of plain values with a ``kind``:

``stateless``  the drop-in operators as the original model code calls them: merge (which plans on every call) and split;
``restore``    merge and split of a scene with the plan in hand (patched attention layers that merge raw tokens);
``branch``     the same with the block's LayerNorm in front and LayerScale + residual behind (per-layer mode);
``attention``  variable-length attention on the packed qkv tensor, with or without the per-key ``log(count)`` bias;
``chain``      selection, plan and a run of frame / global layers launched from Python, one scene per pass;
``graph``      the same for a batch of scenes with a merge ratio per frame, replayed from one CUDA graph;
``direct``     one attention block in per-layer mode with its two projections;
``stack``      the merged forward pass of the alternating-attention stack with all its projections and MLPs.

A frame has 5 special tokens and a patch grid; 37 x 37 patches (a 518 x 518 image, patch 14) is the usual one and 37 x 21 or
28 x 28 are other image formats.  Windows are 3 x 3.  Widths are multiples of the head dimension 64: 1024 (16 heads) is the
usual one, 768 and 384 are the smaller members of the same family of encoders.
"""
from __future__ import annotations

import functools
import math
import random

import torch

from come_b200 import _lib
from come_b200.chain import CoMeOpChain
from come_b200.direct import DirectAttention
from come_b200.flash_attn import flash_attn_varlen_qkvpacked_func, flash_attn_varlen_qkvpacked_func_w_perkey_bias
from come_b200.fused import FusedAggregator
from come_b200.qkv import RotaryPositionEmbedding2D
from come_b200.static_scene import StaticScene
from come_b200.token_merger import MergePlan, func_token_merge_2d, func_token_split, select_windows
from come_b200.vggt_arch import AggregatorCore, Block

START, WINDOW, HEAD_DIM = 5, 3, 64
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
GRIDS = ((37, 37), (37, 28), (37, 21), (28, 28), (36, 36), (21, 37))
CHAIN_LAYERS = 48  # 24 frame / global pairs, the depth of the aggregator
STACK_PAIRS = 4    # block pairs of the stack case: the blocks are alike, four pairs stand for the 24


def listed():
    return [
        # one image, the operators of the drop-in as the unpatched model calls them (float32 features, plan on every call)
        {"name": "stateless_1frame_f32", "kind": "stateless", "frames": 1, "grid_h": 37, "grid_w": 37, "channels": 1024,
         "dtype": "f32", "ratio": 0.5},
        # a long capture: merge and restore 100 frames of float32 features, the largest data movement
        {"name": "restore_100frames_f32", "kind": "restore", "frames": 100, "grid_h": 37, "grid_w": 37, "channels": 1024,
         "dtype": "f32", "ratio": 0.5},
        # an ordinary scene in per-layer mode: LayerNorm + merge in front, LayerScale + residual + split behind
        {"name": "branch_8frames_bf16", "kind": "branch", "frames": 8, "grid_h": 37, "grid_w": 37, "channels": 1024,
         "dtype": "bf16", "ratio": 0.5},
        # frame attention of one landscape image pair: the shortest attention calls of a deployment
        {"name": "attention_2x455_bf16", "kind": "attention", "segments": 2, "shortest": 446, "longest": 455, "heads": 16,
         "dtype": "bf16", "bias": True},
        # a dense encoder block in front of the merge: unmerged frames, no bias, float16
        {"name": "attention_8x1374_f16", "kind": "attention", "segments": 8, "shortest": 1374, "longest": 1374, "heads": 16,
         "dtype": "f16", "bias": False},
        # frame attention of a batch after merging: 64 ragged frames
        {"name": "attention_64ragged_bf16", "kind": "attention", "segments": 64, "shortest": 798, "longest": 1374,
         "heads": 16, "dtype": "bf16", "bias": True},
        # global attention of an 8-frame scene after merging
        {"name": "attention_1x6456_bf16", "kind": "attention", "segments": 1, "shortest": 6456, "longest": 6456, "heads": 16,
         "dtype": "bf16", "bias": True},
        # global attention of a 100-frame scene after merging: the largest single call
        {"name": "attention_1x80672_bf16", "kind": "attention", "segments": 1, "shortest": 80672, "longest": 80672,
         "heads": 16, "dtype": "bf16", "bias": True},
        # a 4-frame scene, all 48 layers launched one by one from Python
        {"name": "chain_4frames_bf16", "kind": "chain", "frames": 4, "grid_h": 37, "grid_w": 37, "heads": 16,
         "dtype": "bf16", "ratio": 0.5, "layers": CHAIN_LAYERS},
        # batch throughput: 8 independent scenes of 4 frames, ragged merge ratios, one CUDA graph of 48 layers
        {"name": "graph_8scenes_of_4_bf16", "kind": "graph", "scenes": 8, "frames": 4, "grid_h": 37, "grid_w": 37,
         "heads": 16, "dtype": "bf16", "ratio_low": 0.25, "ratio_high": 0.75, "layers": CHAIN_LAYERS},
        # one global attention block of an 8-frame scene in per-layer mode, projections included
        {"name": "direct_8frames_global_bf16", "kind": "direct", "frames": 8, "grid_h": 37, "grid_w": 37, "heads": 16,
         "dtype": "bf16", "ratio": 0.5, "global": True},
        # the accelerated stack on an 8-frame scene
        {"name": "stack_8frames_bf16", "kind": "stack", "frames": 8, "grid_h": 37, "grid_w": 37, "dtype": "bf16",
         "ratio": 0.5, "pairs": STACK_PAIRS},
    ]


def _spread(rng: random.Random, low: int, high: int) -> int:
    """Whole number between the bounds, uniform in its logarithm."""
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _grid(rng: random.Random):
    return GRIDS[0] if rng.random() < 0.4 else rng.choice(GRIDS)


def draw(rng: random.Random):
    kind = rng.choice(("stateless", "restore", "branch", "attention", "attention", "attention", "chain", "graph", "direct",
                       "stack"))
    h, w = _grid(rng)
    ratio = round(rng.uniform(0.25, 0.75), 3)
    channels = rng.choice((1024, 1024, 768, 384))
    half = rng.choice(("bf16", "bf16", "f16"))
    if kind in ("stateless", "restore", "branch"):
        return {"kind": kind, "frames": _spread(rng, 1, 16 if kind == "stateless" else 100), "grid_h": h, "grid_w": w,
                "channels": channels, "dtype": rng.choice(("f32", "bf16", "f16")), "ratio": ratio}
    if kind == "attention":
        heads = channels // HEAD_DIM
        form = rng.choice(("frames", "scene", "scene"))
        if form == "frames":
            longest = rng.randint(300, 1374)
            return {"kind": kind, "segments": _spread(rng, 1, 64), "shortest": rng.randint(longest // 2, longest),
                    "longest": longest, "heads": heads, "dtype": half, "bias": rng.random() < 0.75}
        length = _spread(rng, 1000, 60000)
        segments = _spread(rng, 1, max(1, min(8, 60000 // length)))
        return {"kind": kind, "segments": segments, "shortest": length - length // 16, "longest": length, "heads": heads,
                "dtype": half, "bias": rng.random() < 0.75}
    if kind == "chain":
        return {"kind": kind, "frames": _spread(rng, 1, 16), "grid_h": h, "grid_w": w, "heads": channels // HEAD_DIM,
                "dtype": half, "ratio": ratio, "layers": 2 * rng.randint(4, CHAIN_LAYERS // 2)}
    if kind == "graph":
        low = round(rng.uniform(0.2, 0.6), 3)
        return {"kind": kind, "scenes": _spread(rng, 1, 8), "frames": _spread(rng, 1, 8), "grid_h": h, "grid_w": w,
                "heads": channels // HEAD_DIM, "dtype": half, "ratio_low": low, "ratio_high": round(low + 0.2, 3),
                "layers": 2 * rng.randint(4, CHAIN_LAYERS // 2)}
    if kind == "direct":
        return {"kind": kind, "frames": _spread(rng, 1, 24), "grid_h": h, "grid_w": w, "heads": channels // HEAD_DIM,
                "dtype": half, "ratio": ratio, "global": rng.random() < 0.5}
    return {"kind": kind, "frames": _spread(rng, 1, 16), "grid_h": h, "grid_w": w, "dtype": "bf16", "ratio": ratio,
            "pairs": STACK_PAIRS}


# ---------------------------------------------------------------------------------------------------------------
# sizes
# ---------------------------------------------------------------------------------------------------------------
def _tokens(case) -> int:
    return START + case["grid_h"] * case["grid_w"]


def _windows(case) -> int:
    return (case["grid_h"] // WINDOW) * (case["grid_w"] // WINDOW)


def _packed(case, ratio: float) -> int:
    """Packed rows of one frame whose windows are ranked against each other: the merged ones are those below the
    interpolated quantile."""
    return _tokens(case) - (WINDOW * WINDOW - 1) * math.ceil(ratio * (_windows(case) - 1))


def _lengths(case):
    """Segment lengths of an attention case, spread evenly over its range."""
    n, low, high = case["segments"], case["shortest"], case["longest"]
    return [high - (high - low) * ((i * 7) % n) // max(n - 1, 1) for i in range(n)]


def _layout(case):
    return _lib.Layout.two_d(START, case["grid_h"], case["grid_w"], WINDOW, WINDOW)


# ---------------------------------------------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------------------------------------------
def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, shape, dtype):
    return torch.randn(shape, device="cuda", generator=g).to(dtype)


def _mask(case, g, frames, ratio):
    conf = torch.rand((1, frames * case["grid_h"] * case["grid_w"]), device="cuda", generator=g)
    return select_windows(conf, 1, frames, case["grid_h"], case["grid_w"], WINDOW, WINDOW, ratio, "pairwise-rank", "frame")


@functools.lru_cache(maxsize=4)
def _attention_layer(heads: int, is_global: bool, dtype: str):
    """An attention block with fixed random weights: they do not change from scene to scene."""
    torch.manual_seed(1)
    width = heads * HEAD_DIM
    block = Block(width, heads, rope=RotaryPositionEmbedding2D(100.0)).eval().to("cuda", DTYPES[dtype])
    return block, DirectAttention(block.attn, is_global=is_global, run_dtype="fp16" if dtype == "f16" else "bf16").eval()


@functools.lru_cache(maxsize=1)
def _stack(pairs: int, dtype: str):
    core = AggregatorCore(depth=pairs, retain_layers=frozenset({pairs // 2 - 1, pairs - 1})).to("cuda", DTYPES[dtype])
    return FusedAggregator(core).eval()


def prepare(case, seed):
    kind, g = case["kind"], _generator(seed)
    dtype = DTYPES[case["dtype"]]
    state = {"case": case}
    if kind in ("stateless", "restore", "branch"):
        frames, n, c = case["frames"], _tokens(case), case["channels"]
        state["x"] = _normal(g, (frames, n, c), dtype)
        state["mask"] = _mask(case, g, frames, case["ratio"])
        if kind != "stateless":
            state["plan"] = MergePlan(state["mask"], _layout(case))
        if kind == "branch":
            norm = torch.nn.LayerNorm(c, eps=1e-6).to("cuda", dtype)
            with torch.no_grad():
                norm.weight.copy_(1.0 + 0.1 * torch.randn(c, device="cuda", generator=g))
                norm.bias.copy_(0.02 * torch.randn(c, device="cuda", generator=g))
            state["norm"] = norm
            state["scale"] = _normal(g, (c,), dtype) * 0.01
    elif kind == "attention":
        lengths = _lengths(case)
        total = sum(lengths)
        ends = [0]
        for n in lengths:
            ends.append(ends[-1] + n)
        state["cu"] = torch.tensor(ends, dtype=torch.int32, device="cuda")
        state["longest"] = max(lengths)
        state["qkv"] = _normal(g, (total, 3, case["heads"], HEAD_DIM), dtype)
        # about a tenth of the rows of a half-merged frame stand for a 3 x 3 window
        state["bias"] = torch.where(torch.rand(total, device="cuda", generator=g) < 0.1, 9.0, 1.0).log().to(dtype)
    elif kind == "chain":
        frames, h, w, heads = case["frames"], case["grid_h"], case["grid_w"], case["heads"]
        state["chain"] = CoMeOpChain(frames, START, h, w, WINDOW, WINDOW, case["ratio"], heads, HEAD_DIM,
                                     ["frame", "global"] * (case["layers"] // 2))
        state["x"] = _normal(g, (frames, _tokens(case), heads * HEAD_DIM), dtype)
        state["conf"] = torch.rand((1, frames * h * w), device="cuda", generator=g)
        state["qkv"] = _normal(g, (frames * _tokens(case), 3, heads, HEAD_DIM), dtype)
    elif kind == "graph":
        scenes, fps, h, w, heads = case["scenes"], case["frames"], case["grid_h"], case["grid_w"], case["heads"]
        frames, n = scenes * fps, _tokens(case)
        scene = StaticScene(frames, heads * HEAD_DIM, START, h, w, WINDOW, WINDOW, 0.5, heads, HEAD_DIM,
                            ["frame", "global"] * (case["layers"] // 2), "frame", dtype, torch.device("cuda", 0), fps, True)
        span = case["ratio_high"] - case["ratio_low"]
        scene.ratios.copy_(case["ratio_low"] + span * torch.rand(frames, device="cuda", generator=g))
        state["x"] = _normal(g, (frames, n, heads * HEAD_DIM), dtype)
        state["conf"] = torch.rand((scenes, fps * h * w), device="cuda", generator=g).to(dtype)
        state["qkv"] = _normal(g, (frames * n, 3, heads, HEAD_DIM), dtype)
        scene.x.copy_(state["x"])  # the capture runs the sequence once: on a scene, not on uninitialised memory
        scene.conf.copy_(state["conf"])
        scene.qkv.copy_(state["qkv"])
        state["scene"] = scene.capture()
    elif kind == "direct":
        frames, heads, n = case["frames"], case["heads"], _tokens(case)
        state["block"], state["layer"] = _attention_layer(heads, case["global"], case["dtype"])
        x = _normal(g, (frames, n, heads * HEAD_DIM), dtype)
        state["x"] = x.reshape(1, frames * n, -1) if case["global"] else x
        state["plan"] = MergePlan(_mask(case, g, frames, case["ratio"]), _layout(case))
        state["plan"].positions()
    else:
        frames = case["frames"]
        state["model"] = _stack(case["pairs"], case["dtype"])
        state["x"] = _normal(g, (1, frames, _tokens(case), 1024), dtype)
        state["plan"] = MergePlan(_mask(case, g, frames, case["ratio"]), _layout(case))
    return state


# ---------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "stateless":
        x = state["x"]
        frames, n, c = x.shape
        jagged, rev = func_token_merge_2d(x, START, WINDOW, WINDOW, case["grid_h"], case["grid_w"], state["mask"],
                                          allow_ragged=True)
        return jagged.tokens, jagged.weight, jagged.offset, rev, func_token_split(jagged, rev, (1, frames, n, c))
    if kind == "restore":
        merged = state["plan"].merge(state["x"])
        return merged, state["plan"].split(merged)
    if kind == "branch":
        merged = state["plan"].merge_layernorm(state["x"], state["norm"])
        return merged, state["plan"].split_add(merged, state["x"], state["scale"])
    if kind == "attention":
        scale = HEAD_DIM ** -0.5
        if case["bias"]:
            return flash_attn_varlen_qkvpacked_func_w_perkey_bias(state["qkv"], state["cu"], state["longest"], state["bias"],
                                                                  softmax_scale=scale)
        return flash_attn_varlen_qkvpacked_func(state["qkv"], state["cu"], state["longest"], softmax_scale=scale)
    if kind == "chain":
        chain = state["chain"]
        plan = chain.build_plan(state["conf"])
        qkv = state["qkv"][: plan.total]
        last = {}
        for name in chain.layer_kinds:
            last[name] = chain.layer(plan, state["x"], qkv, name)
        return plan.offset, plan.rev_id, last["frame"], last["global"]
    if kind == "graph":
        return state["scene"].run(state["x"], state["conf"], state["qkv"])
    with torch.no_grad():
        if kind == "direct":
            block = state["block"]
            return state["layer"].forward_residual(state["x"], state["plan"], case["frames"], block.norm1, block.ls1.gamma)
        out, _ = state["model"](state["x"], state["plan"])
        return out


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exact its results are
# ---------------------------------------------------------------------------------------------------------------
def work(case):
    kind, e = case["kind"], 4 if case["dtype"] == "f32" else 2
    if kind == "attention":
        lengths = _lengths(case)
        width = case["heads"] * HEAD_DIM
        return {"bytes": sum(lengths) * (4 * width + case["bias"]) * e, "flops": sum(4.0 * n * n * width for n in lengths)}
    frames = case["frames"] * case.get("scenes", 1)
    n = _tokens(case)
    p = _packed(case, case["ratio"] if "ratio" in case else 0.5 * (case["ratio_low"] + case["ratio_high"]))
    dense, packed = frames * n, frames * p
    if kind in ("stateless", "restore", "branch"):
        c = case["channels"]
        rows = dense + packed + packed + dense + (dense if kind == "branch" else 0)
        return {"bytes": rows * c * e + dense * 8 + frames * _windows(case), "flops": 2.0 * dense * c}
    width = case["heads"] * HEAD_DIM if kind != "stack" else 1024
    frame_flops, scene_flops = 4.0 * p * packed * width, 4.0 * packed * (packed / case.get("scenes", 1)) * width
    if kind in ("chain", "graph"):
        layer = (2 * dense + 6 * packed) * width * e + dense * 8  # merge, attention (qkv in, out), restore
        return {"bytes": case["layers"] * layer, "flops": case["layers"] / 2 * (frame_flops + scene_flops)}
    if kind == "direct":
        return {"bytes": (3 * dense + 10 * packed) * width * e + 4 * width * width * e,
                "flops": 8.0 * packed * width * width + (scene_flops if case["global"] else frame_flops)}
    blocks = 2 * case["pairs"]
    return {"bytes": (dense + 4 * dense + blocks * 26 * packed) * width * e + blocks * 12 * width * width * e,
            "flops": blocks * 24.0 * packed * width * width + case["pairs"] * (frame_flops + scene_flops)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("stateless", "restore"):
        # means of 9 values summed in float32; one rounding to the element type
        return {"rel": 1e-6 if case["dtype"] == "f32" else 1e-3}
    if kind == "branch":
        return {"rel": 1e-5 if case["dtype"] == "f32" else 5e-3}
    if kind == "direct":
        return {"rel": 3e-3}  # a scaled branch added to a 16-bit stream: the rounding of the stream
    return {"rel": 1e-2}  # probabilities and outputs in 16 bits
