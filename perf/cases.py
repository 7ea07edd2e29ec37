"""Performance cases of the MoE block: what a user of this library has it do, through its public entry points.

One layer shape, the one the repository's configurations name (hidden 2048, 256 experts, top-8, expert and shared
intermediate 512, dense fp16 router, scalar shared-expert gate), in the four ways it is driven:

  token    a decoder's loop over its layers, one or two rows (plain decoding, two-row verification): per layer the block
           with the residual add and norm before it and the next block's input norm after it
  stack    a whole stack of MoE blocks in one call, one to eight rows
  batch    one block for a decode batch of independent rows
  prefill  one block for a chunk of a prompt

Weights and rows are synthetic and made on the device from the seed.
"""
from __future__ import annotations

import numpy as np
import torch

from nvmai_b200 import MoE, MoEConfig, synthetic
from nvmai_b200 import format as fmt

D, F, E, K = 2048, 512, 256, 8
EPS = 1e-6
LEAN = 2.0          # see _lean
META = {"bf16": fmt.META_BF16, "fp16": fmt.META_FP16}
OUT = {"fp16": fmt.OUT_FP16, "fp32": fmt.OUT_FP32}
OUT_TORCH = {"fp16": torch.float16, "fp32": torch.float32}


def _case(kind, rows, bits, *, layers=1, meta="bf16", out="fp16", skew=0.0, lean=0.0):
    return {"kind": kind, "rows": rows, "bits": bits, "layers": layers, "meta": meta, "out": out, "skew": skew,
            "lean": lean}


def listed():
    named = [
        # plain decoding of one stream: eight layers of a decoder's loop, the smallest calls there are
        ("token_1row_4bit", _case("token", 1, 4, layers=8)),
        # verification of one speculated token: the same loop with two rows, 8-bit experts
        ("token_2rows_8bit", _case("token", 2, 8, layers=8)),
        # the benchmark's workload: the 40-layer stack, one row, both weight formats
        ("stack_1row_4bit", _case("stack", 1, 4, layers=40, out="fp32", lean=LEAN)),
        ("stack_1row_8bit", _case("stack", 1, 8, layers=40, out="fp32", lean=LEAN)),
        # a few streams (or speculated tokens) decoded together through one call
        ("stack_5rows_4bit", _case("stack", 5, 4, layers=4, out="fp32")),
        # small decode batches of independent rows
        ("batch_4rows_8bit", _case("batch", 4, 8, meta="fp16", out="fp32")),
        ("batch_13rows_4bit", _case("batch", 13, 4)),
        # serving: tens to hundreds of rows, uniform and with a few popular experts
        ("batch_64rows_8bit", _case("batch", 64, 8)),
        ("batch_256rows_4bit_skewed", _case("batch", 256, 4, out="fp32", skew=1.1)),
        # prompts: a short ragged one, a ragged 8-bit chunk, the benchmark's full chunk
        ("prefill_201rows_4bit", _case("prefill", 201, 4, skew=0.6)),
        ("prefill_1531rows_8bit", _case("prefill", 1531, 8)),
        ("prefill_4096rows_4bit", _case("prefill", 4096, 4)),
    ]
    return [dict(c, name=name) for name, c in named]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("token", "stack", "batch", "batch", "prefill", "prefill"))
    bits = rng.choice((4, 8))
    meta = rng.choice(("bf16", "bf16", "fp16"))
    out = rng.choice(("fp16", "fp32"))
    if kind == "token":
        return _case(kind, rng.choice((1, 1, 2)), bits, layers=rng.randint(3, 24), meta=meta, out=out)
    if kind == "stack":
        if rng.random() < 0.5:
            return _case(kind, 1, bits, layers=_log_int(rng, 6, 40), out="fp32", lean=LEAN)
        return _case(kind, rng.randint(2, 8), bits, layers=rng.randint(2, 4), meta=meta, out=out)
    skew = rng.choice((0.0, 0.0, round(rng.uniform(0.3, 1.2), 2)))
    if kind == "batch":
        return _case(kind, _log_int(rng, 3, 256), bits, meta=meta, out=out, skew=skew)
    return _case(kind, _log_int(rng, 32, 4096 if bits == 4 else 2600), bits, meta=meta, out=out, skew=skew)


def _lean(dev, lean):
    """Gives the weights a common mean, in units in which 1.0 makes the mean of a dot product with a constant row as
    large as its spread.  A deep chain of blocks without residuals then settles (the rounding of a layer fades); around
    zero-mean weights every layer multiplies what came before by about 1.4."""
    def shift(biases, n):
        biases += lean * 0.0575 / n ** 0.5
    off, experts = dev["offsets"], dev["experts"]
    for name, n in (("gate", D), ("up", D), ("down", F)):
        start = off[name + "_b"]
        shift(experts[:, start:start + D * F // fmt.GROUP * 2].view(dev["shared"][0][2].dtype), n)
    for (_, _, biases), n in zip(dev["shared"], (D, D, F)):
        shift(biases, n)


def _layer(case, seed):
    """One layer's weights on the device; `skew` > 0: the router prefers experts about as 1 / rank^skew."""
    dev = synthetic.device_layer(seed, d=D, f=F, shared_f=F, num_experts=E, routed_bits=case["bits"],
                                 shared_bits=case["bits"], meta=META[case["meta"]])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 1)
    if case["lean"]:
        _lean(dev, case["lean"])
    if case["skew"]:
        # the rows share a component along one direction (_rows), and each router row answers to it by the logarithm of
        # its expert's popularity
        rank = torch.randperm(E, device="cuda", generator=gen).float() + 1.0
        bias = -case["skew"] * torch.log(rank)
        router = dev["router"][0].float() + bias[:, None] * _direction()[None, :] / 8.0
        dev["router"] = (router.to(torch.float16), None, None)
    return dev


def _direction():
    sign = 1.0 - 2.0 * (torch.arange(D, device="cuda") % 2).float()
    return sign / D ** 0.5


def _rows(case, count, gen, std=1.0):
    x = torch.randn((count, D), device="cuda", generator=gen) * std
    if case["skew"]:
        x += 8.0 * std * _direction()
    return x


class State:
    pass


def prepare(case, seed):
    rows, layers = case["rows"], case["layers"]
    s = State()
    s.case = case
    cfg = MoEConfig(d=D, f=F, shared_f=F, num_experts=E, top_k=K, routed_bits=case["bits"], shared_bits=case["bits"],
                    router_kind=fmt.ROUTER_DENSE_F16, shared_gate_kind=fmt.ROUTER_DENSE_F16,
                    meta_dtype=META[case["meta"]], activation=fmt.ACT_SILU, out_dtype=OUT[case["out"]],
                    max_tokens=rows, num_layers=layers)
    s.moe = MoE(cfg)
    s.weights = [_layer(case, 1000 * seed + 2 * l) for l in range(layers)]
    for l, dev in enumerate(s.weights):
        synthetic.register_device_layer(s.moe, l, dev)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000 * seed + 999)
    out = OUT_TORCH[case["out"]]
    s.stream = torch.cuda.current_stream()
    if case["kind"] == "token":
        # a residual stream is much larger than what one block adds to it
        s.embed = _rows(case, rows, gen, 32.0).to(out)
        s.hidden = s.embed.clone()
        s.delta = [_rows(case, rows, gen).to(torch.float16) for _ in range(layers)]
        s.norm = [(torch.rand(D, device="cuda", generator=gen) * 0.5 + 0.75).to(torch.bfloat16) for _ in range(layers)]
        s.next_norm = [(torch.rand(D, device="cuda", generator=gen) * 0.5 + 0.75).to(torch.bfloat16) for _ in range(layers)]
        s.x_next = torch.empty((layers, rows, D), dtype=torch.float16, device="cuda")
    else:
        s.x = _rows(case, rows, gen).to(torch.float16)
        s.y = torch.empty((rows, D), dtype=out, device="cuda")
    if case["kind"] in ("batch", "prefill"):
        s.idx = torch.empty((rows, K), dtype=torch.int32, device="cuda")
        s.w = torch.empty((rows, K), dtype=torch.float16, device="cuda")
        s.hidden = _rows(case, rows, gen, 32.0).to(out)
    return s


def run(s):
    kind, rows = s.case["kind"], s.case["rows"]
    if kind == "token":
        s.hidden.copy_(s.embed)               # the token's embedding enters the residual stream
        for l in range(s.case["layers"]):
            s.moe.layer_decode_fused_norms(l, s.hidden, s.norm[l], EPS, rows, s.next_norm[l], EPS, s.x_next[l],
                                           attn_delta=s.delta[l], stream=s.stream)
        return s.hidden, s.x_next
    if kind == "stack":
        s.moe.stack_decode(s.x, rows, s.y, stream=s.stream)
        return s.y
    if kind == "batch":
        s.moe.layer_decode(0, s.x, rows, hidden=s.hidden, h2_out=s.y, out_idx=s.idx, out_w=s.w, stream=s.stream)
        return s.hidden, s.y, s.idx, s.w
    s.moe.layer_prefill(0, s.x, rows, hidden=s.hidden, out_idx=s.idx, out_w=s.w, stream=s.stream)
    return s.hidden, s.idx, s.w


def _distinct_experts(case):
    """Experts that the rows of one layer select, on average (drawn once from the logits' distribution)."""
    if case["rows"] == 1:
        return K
    r = np.random.default_rng(1)
    logits = r.normal(0.0, 0.02 * D ** 0.5, size=(case["rows"], E)) - case["skew"] * np.log(np.arange(E) + 1.0)
    return len(np.unique(np.argpartition(-logits, K, axis=1)[:, :K]))


def work(case):
    """Each selected expert's weights once, the shared expert, the router and the gate row; rows in and out."""
    rows, layers, bits = case["rows"], case["layers"], case["bits"]
    expert = 3 * (D * F * bits // 8 + 2 * (D * F // fmt.GROUP) * 2)
    weights = (_distinct_experts(case) + 1) * expert + (E + 1) * D * 2
    out = rows * D * (2 if case["out"] == "fp16" else 4)
    if case["kind"] == "token":              # delta and norm weights in, x_next out, per layer; hidden in and out
        nbytes = layers * (weights + 2 * rows * D * 2 + 2 * D * 2) + 2 * out
    elif case["kind"] == "stack":
        nbytes = layers * weights + rows * D * 2 + out
    else:                                    # x in, hidden in and out, routing out, and the batch's block output
        nbytes = weights + rows * D * 2 + 2 * out + rows * K * 6 + (out if case["kind"] == "batch" else 0)
    return {"bytes": nbytes, "flops": layers * rows * 2 * ((K + 1) * 3 * D * F + (E + 1) * D)}


def tolerance(case):
    # 11-bit activations and outputs; a chain of blocks carries the rounding of each layer into the next, and a leaning
    # one lets it fade
    if case["lean"]:
        return {"rel": 3e-3}
    if case["kind"] in ("token", "stack"):
        return {"rel": 1e-2}
    return {"rel": 2e-3, "max": 0.05, "differ": 2e-3}
