"""The work that a user of this library has it do, as cases that can be timed.

Five kinds of pass, each through the public entry point a serving program calls:

  block  one MoeBlock.forward on device rows (a layer between a caller's own mixers)
  stack  the 40 MoE layers of a decode step: rows in, one captured graph, hidden state out (MoeStack.run)
  host   one MoeBlock.forward_host on pinned host rows
  dense  one DenseFfnBlock.forward of the 27B sibling (hidden 5120, intermediate 17408)
  head   logits over the 248,320-entry vocabulary and their argmax (LmHeadKernels.forward, .argmax)

The MoE layer is the 256-expert, top-8, hidden 2048, intermediate 512 geometry.  `tokens` are live,
`width` is what the handle was made for (a server makes its handles once and runs ragged batches on
them).  `layout` says how the tensors are quantised:

  q6_k     everything Q6_K (the benchmark's default)
  mixed    Q6_K experts, Q8_0 shared expert (the 40-layer benchmark stack)
  shipped  Q6_K gate and up, Q8_0 down and shared expert (a UD-Q6_K_XL file)
  q8_0     everything Q8_0
"""
from __future__ import annotations

import math

import numpy as np
import torch

from llmxabe_b200.lm_head import HeadFormat, HeadTensor, LmHeadGeometry, LmHeadKernels
from llmxabe_b200.moe import (DenseFfnBlock, ExpertQuant, MoeBlock, MoeGeometry, MoeLayerWeights, QuantTensor,
                              moe_block_size)
from llmxabe_b200.stack import MoeStack
from llmxabe_b200.synth import zipf_bias

E, K, H, I = 256, 8, 2048, 512
DENSE_H, DENSE_I = 5120, 17408
LAYERS = 40
VOCAB = 248_320

Q6, Q8 = ExpertQuant.Q6K, ExpertQuant.Q8_0
# layout -> formats of (routed gate and up, routed down, shared expert)
LAYOUTS = {"q6_k": (Q6, Q6, Q6), "mixed": (Q6, Q6, Q8), "shipped": (Q6, Q8, Q8), "q8_0": (Q8, Q8, Q8)}

# A trained matrix of this family has entries of about 0.02: the super-block scale that gives it, from the
# rms of what it multiplies (6-bit codes 18.5 times int8 scales in [-32, 31] 18.5; int8 codes 73.9).
WEIGHT_STD = 0.02
SCALE = {Q6: WEIGHT_STD / (18.5 * 18.5), Q8: WEIGHT_STD / 73.9}


def listed():
    return [
        # one token through one layer, launched by the caller: what a call costs at least
        {"name": "block_1", "kind": "block", "tokens": 1, "width": 1, "layout": "q6_k", "dtype": "f32"},
        # one sequence being decoded
        {"name": "stack_1", "kind": "stack", "tokens": 1, "width": 1, "layout": "mixed"},
        # a server's decode step with a batch that fills its bucket only in part, tensors as shipped
        {"name": "stack_19_of_32", "kind": "stack", "tokens": 19, "width": 32, "layout": "shipped"},
        # 64 concurrent sequences: the headline decode
        {"name": "stack_64", "kind": "stack", "tokens": 64, "width": 64, "layout": "q6_k"},
        # the same batch handed over in host memory
        {"name": "host_64", "kind": "host", "tokens": 64, "width": 64, "layout": "mixed"},
        # a short prompt, or a prompt's last piece
        {"name": "block_333_of_384", "kind": "block", "tokens": 333, "width": 384, "layout": "mixed", "dtype": "bf16"},
        # one prefill chunk with bf16 rows
        {"name": "block_2048", "kind": "block", "tokens": 2048, "width": 2048, "layout": "q6_k", "dtype": "bf16"},
        # the largest prefill batch
        {"name": "block_16384", "kind": "block", "tokens": 16384, "width": 16384, "layout": "mixed", "dtype": "f32"},
        # the dense sibling: one sequence, a ragged decode batch, a prefill chunk
        {"name": "dense_1", "kind": "dense", "tokens": 1, "width": 1, "layout": "q6_k"},
        {"name": "dense_43_of_64", "kind": "dense", "tokens": 43, "width": 64, "layout": "q6_k"},
        {"name": "dense_4096", "kind": "dense", "tokens": 4096, "width": 4096, "layout": "q6_k"},
        # greedy sampling for three concurrent sequences
        {"name": "head_3", "kind": "head", "tokens": 3, "width": 8, "layout": "q8_0"},
    ]


def _log_between(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)) - 1e-9)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "stack", "stack", "host", "dense", "dense", "head"])
    most = {"block": 16384, "stack": 64, "host": 64, "dense": 4096, "head": 64}[kind]
    tokens = _log_between(rng, 2, most)  # one token is listed for the kinds where it matters most
    # a handle made for just this batch, a power-of-two bucket, or some other limit that the batch stays under
    width = rng.choice([tokens, 1 << (tokens - 1).bit_length(), rng.randint(tokens, 2 * tokens + 6)])
    case = {"kind": kind, "tokens": tokens, "width": min(width, most)}
    if kind == "head":
        case["layout"] = rng.choice(["q8_0", "q8_0", "q6_k"])
    elif kind == "dense":
        case["layout"] = rng.choice(["q6_k", "q6_k", "q8_0"])
    else:
        case["layout"] = rng.choice(["q6_k", "mixed", "mixed", "shipped", "shipped", "q8_0"])
    if kind == "block":
        case["dtype"] = rng.choice(["f32", "bf16"])
    return case


# ---------------------------------------------------------------- inputs
def _quant_tensor(quant, count, gen):
    """`count` weights in GGUF file layout: uniform codes, half-normal super-block scales."""
    dev = gen.device
    per, size = quant.block_elements, quant.file_block_bytes
    blocks = count // per
    out = torch.randint(0, 256, (blocks, size), dtype=torch.uint8, device=dev, generator=gen)
    d = (torch.randn(blocks, device=dev, generator=gen).abs() * SCALE[quant]).to(torch.float16)
    d = d.view(torch.uint8).view(blocks, 2)
    if quant is Q6:
        out[:, 192:208] = torch.randint(-32, 32, (blocks, 16), dtype=torch.int8, device=dev,
                                        generator=gen).view(torch.uint8)
        out[:, 208:210] = d
    else:
        out[:, 0:2] = d
    return out.view(-1)


def _moe_layer(layout, seed, layer, skewed, gen):
    routed, down, shared = LAYOUTS[layout]
    n = E * I * H
    q = lambda quant, count: _quant_tensor(quant, count, gen)
    return MoeLayerWeights(
        layer=layer, post_norm=1 + 0.1 * torch.randn(H, device=gen.device, generator=gen),
        router=torch.randn(E, H, device=gen.device, generator=gen) * 0.02,
        router_bias=torch.from_numpy(zipf_bias(E, seed, layer)) if skewed else None,
        gate_exps=q(routed, n), gate_quant=routed, up_exps=q(routed, n), up_quant=routed,
        down_exps=q(down, n), down_quant=down,
        shared_gate_inp=torch.randn(H, device=gen.device, generator=gen) * 0.02,
        shared_gate=q(shared, I * H), shared_gate_quant=shared, shared_up=q(shared, I * H), shared_up_quant=shared,
        shared_down=q(shared, I * H), shared_down_quant=shared, device=gen.device)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, tokens, width, layout = case["kind"], case["tokens"], case["width"], case["layout"]
    rows = lambda n, h: torch.randn(n, h, device="cuda", generator=gen)
    if kind == "head":
        geometry = LmHeadGeometry(H, VOCAB, width)
        fmt = HeadFormat.Q8_0 if layout == "q8_0" else HeadFormat.Q6K
        weight = HeadTensor(_quant_tensor(ExpertQuant(int(fmt)), geometry.elements(), gen), fmt)
        return dict(kind=kind, tokens=tokens, head=LmHeadKernels(geometry), weight=weight, x=rows(width, H),
                    logits=torch.zeros(width, VOCAB, device="cuda"),
                    best=torch.zeros(width, dtype=torch.int32, device="cuda"))
    if kind == "dense":
        quant = LAYOUTS[layout][0]
        n = DENSE_H * DENSE_I
        w = [QuantTensor(_quant_tensor(quant, n, gen), quant) for _ in range(3)]
        geometry = MoeGeometry.qwen3_8_27b_dense(moe_block_size(width), width)
        return dict(kind=kind, tokens=tokens, block=DenseFfnBlock(geometry), w=w,
                    post_norm=1 + 0.1 * torch.randn(DENSE_H, device="cuda", generator=gen),
                    x=rows(width, DENSE_H), ffn_out=torch.zeros(width, DENSE_H, device="cuda"),
                    l_out=torch.zeros(width, DENSE_H, device="cuda"))
    geometry = MoeGeometry.qwen3_6(moe_block_size(width), width)
    skewed = tokens > 1  # of many tokens, some experts get more than others
    if kind == "stack":
        layers = [_moe_layer(layout, seed, i, skewed, gen) for i in range(LAYERS)]
        stack = MoeStack(geometry, layers)
        x = rows(tokens, H)
        stack.run(x)
        stack.capture()
        return dict(kind=kind, stack=stack, x=x)
    w = _moe_layer(layout, seed, 0, skewed, gen)
    state = dict(kind=kind, tokens=tokens, block=MoeBlock(geometry), w=w)
    if kind == "host":
        pinned = lambda: torch.zeros(width, H, pin_memory=True)
        state.update(x=pinned(), ffn_out=pinned(), l_out=pinned())
        state["x"].copy_(rows(width, H))
    else:
        x = rows(width, H)
        state.update(x=x.bfloat16() if case["dtype"] == "bf16" else x, ffn_out=torch.zeros(width, H, device="cuda"),
                     l_out=torch.zeros(width, H, device="cuda"))
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    kind, s = state["kind"], state
    if kind == "stack":
        return s["stack"].run(s["x"])
    t = s["tokens"]
    if kind == "head":
        s["head"].forward(s["weight"], s["x"], t, s["logits"])
        s["head"].argmax(s["logits"], t, s["best"])
        return {"logits": s["logits"][:t], "argmax": s["best"][:t]}
    if kind == "dense":
        s["block"].forward(s["post_norm"], *s["w"], s["x"], t, s["ffn_out"], s["l_out"])
    elif kind == "host":
        s["block"].forward_host(s["w"], s["x"], t, s["ffn_out"], s["l_out"])
    else:
        s["block"].forward(s["w"], s["x"], t, s["ffn_out"], s["l_out"])
    return {"ffn_out": s["ffn_out"][:t], "l_out": s["l_out"][:t]}


# ---------------------------------------------------------------- what a pass cannot do without
def _matrix_bytes(quant, count):
    return count // quant.block_elements * quant.file_block_bytes


def _distinct_experts(tokens):
    """How many of the experts a batch reaches: the router's logits are normal, with the skew's bias on top."""
    t = min(tokens, 4096)
    r = np.random.default_rng(7)
    logits = r.standard_normal((t, E)) * 0.02 * math.sqrt(H) + (zipf_bias(E, 7, 0) if tokens > 1 else 0)
    return len(np.unique(np.argpartition(-logits, K, axis=1)[:, :K]))


def work(case):
    kind, t = case["kind"], case["tokens"]
    if kind == "head":
        quant = Q8 if case["layout"] == "q8_0" else Q6
        return {"bytes": _matrix_bytes(quant, VOCAB * H) + t * 4 * (H + VOCAB + 1), "flops": 2 * t * VOCAB * H}
    if kind == "dense":
        n = DENSE_H * DENSE_I
        return {"bytes": 3 * _matrix_bytes(LAYOUTS[case["layout"]][0], n) + 4 * DENSE_H * (1 + 3 * t),
                "flops": 6 * t * n}
    routed, down, shared = LAYOUTS[case["layout"]]
    n = H * I
    weights = (_distinct_experts(t) * (2 * _matrix_bytes(routed, n) + _matrix_bytes(down, n))
               + 3 * _matrix_bytes(shared, n) + 4 * (E * H + 2 * H))
    flops = 2 * t * (3 * n * (K + 1) + E * H)
    if kind == "stack":  # the hidden state goes in once and comes out once
        return {"bytes": LAYERS * weights + 2 * 4 * t * H, "flops": LAYERS * flops}
    row_in = 2 if case.get("dtype") == "bf16" else 4
    return {"bytes": weights + t * H * (row_in + 8), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "head":  # exact codes times activations carried in two f16 parts, summed in fp32
        return {"rel": 1e-5}
    if kind == "stack":  # 40 layers; a near-tie in a late router may fall the other way for a row
        return {"rel": 5e-3}
    return {"rel": 2e-3}  # f16 activations, intermediates and (prefill) weights, fp32 sums: 1e-3 to either side
