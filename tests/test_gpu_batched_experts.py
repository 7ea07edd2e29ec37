"""Edges of the batched experts' kernels (accumulator switches, ragged items, odd K-block counts, scale types) through
the C ABI against the oracle."""
import functools
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
for p_ in (ROOT, ROOT / "tests"):
    if str(p_) not in sys.path:
        sys.path.insert(0, str(p_))

pytestmark = pytest.mark.gpu

from nvmai_b200 import MoE, MoEConfig, synthetic      # noqa: E402
from nvmai_b200 import format as fmt                  # noqa: E402
from oracle import oracle as orc                      # noqa: E402
import gpu_util as gu                                 # noqa: E402

BF16, FP16 = fmt.META_BF16, fmt.META_FP16


def _tol(meta, out, entry):
    """fp32 outputs: a few of a row's activations a half-ulp (2^-11) apart; fp16 outputs: activations, partials and the output
    rounded to half on both sides (2^-11 each, now and then on the other side of a tie); fp16 scales on the prefill entry's
    tcgen05 path round once more in either projection (2^-11 of a weight each): 4 x 2^-11 in all."""
    if meta == FP16 and entry == "prefill":
        return 2e-3
    return 1e-3 if out == fmt.OUT_FP16 else 2e-4


@functools.lru_cache(maxsize=1)      # (0.9 GB at the benchmark's shape)
def _host_layer(seed, bits, meta, d, f, experts, shared_f=None, shared_bits=None):
    """A layer on the host; 8-bit weights zero-mean: the one-sided ones leave fp16's range."""
    shared_f, shared_bits = f if shared_f is None else shared_f, bits if shared_bits is None else shared_bits
    host = synthetic.layer(seed, d=d, f=f, shared_f=shared_f, num_experts=experts, routed_bits=bits, shared_bits=shared_bits, meta=meta)
    if bits == 8:
        rng = np.random.default_rng(seed)
        off = host["offsets"]
        for name, n in (("gate", f * d), ("up", f * d), ("down", d * f)):
            s = rng.uniform(0.0003, 0.0012, size=(experts, n // 64)).astype(np.float32)
            for key, v in (("_s", s), ("_b", -127.5 * s)):
                raw = np.ascontiguousarray(fmt.f32_to_meta_bits(v, meta)).view(np.uint8)
                host["experts"][:, off[name + key]:off[name + key] + raw.shape[1]] = raw
    if shared_bits == 8:
        host["shared"] = [(w, fmt.f32_to_meta_bits(np.full(s.shape, 0.0007), meta), fmt.f32_to_meta_bits(np.full(s.shape, -0.0892), meta))
                          for w, s, _ in host["shared"]]
    return host


def _worst_error(host, cfg, entry, tokens, sample):
    """One call of the entry point; the sampled rows against the oracle."""
    moe = MoE(cfg)
    dl = gu.DeviceLayer(host)
    dl.register(moe, 0)
    x = synthetic.hidden_rows(701, tokens, cfg.d)
    f16 = cfg.out_dtype == fmt.OUT_FP16
    y = gu.dev_empty(tokens * cfg.d, "f16" if f16 else "f32")
    call = moe.layer_decode if entry == "decode" else moe.layer_prefill
    call(0, gu.to_dev(x), tokens, **{"h2_out" if entry == "decode" else "y_out": y})
    moe.synchronize()
    got = (orc.f16_bits_to_f32(gu.from_dev(y, np.uint16)) if f16 else y.cpu().numpy()).reshape(tokens, cfg.d)
    L, keep = gu.oracle_layer(host, cfg)
    worst = 0.0
    for t in sample:
        xr = np.ascontiguousarray(x[t])
        want = gu.oracle_decode(L, cfg, xr)[2] if entry == "decode" else gu.oracle_prefill_row(L, cfg, xr, None)[2]
        worst = max(worst, orc.rel_error(got[t], want))
    return worst


# 8 experts: every expert gets every row, so `tokens` is the experts' row count.  96 / 97 and 192 / 193 rows: where an
# item is split; 16 / 17: one and two 16-row pieces; 1: the smallest item.  f = 384: an odd number of chunks of codes
# per down tile (4-bit), an odd number of A slots per tile; d = 768: 12 K blocks, scales that do not come eight at a time.
@pytest.mark.parametrize("bits,meta,out,tokens,d,f", [
    (4, BF16, fmt.OUT_FP16, 1, 256, 128), (4, BF16, fmt.OUT_FP16, 17, 768, 384), (4, BF16, fmt.OUT_FP32, 96, 256, 384),
    (4, BF16, fmt.OUT_FP16, 97, 512, 128), (4, BF16, fmt.OUT_FP16, 193, 256, 128), (8, BF16, fmt.OUT_FP16, 16, 768, 128),
    (8, BF16, fmt.OUT_FP32, 130, 256, 384), (4, FP16, fmt.OUT_FP16, 33, 768, 384), (8, FP16, fmt.OUT_FP32, 40, 256, 128),
    (8, FP16, fmt.OUT_FP16, 65, 512, 384), (4, BF16, fmt.OUT_FP32, 5, 2048, 512), (8, FP16, fmt.OUT_FP16, 3, 2048, 512)])
@pytest.mark.parametrize("entry", ["decode", "prefill"])
@pytest.mark.parametrize("stream_rows", [0, 1000])
def test_rows_of_every_item_match_the_oracle(bits, meta, out, tokens, d, f, stream_rows, entry, monkeypatch):
    monkeypatch.setenv("NVMAI_CUDA_TC_MIN", "1")
    monkeypatch.setenv("NVMAI_CUDA_STREAM_ROWS", str(stream_rows))     # the tcgen05 kernel, the streaming kernel
    host = _host_layer(700 + tokens, bits, meta, d, f, 8)
    cfg = MoEConfig(d=d, f=f, shared_f=f, num_experts=8, top_k=8, routed_bits=bits, shared_bits=bits, meta_dtype=meta,
                    out_dtype=out, max_tokens=tokens)
    sample = sorted({0, tokens // 2, tokens - 1, min(tokens - 1, 15), min(tokens - 1, 95), min(tokens - 1, 96)})
    assert _worst_error(host, cfg, entry, tokens, sample) < _tol(meta, out, entry)


# Mixed calls: experts with more rows than the limit through the grouped GEMMs, the others (and, where those are few, all
# of them and the shared expert) through the streaming kernel.  40 rows on 32 experts: 10 rows each on average; a limit
# of 8: many above it; 16: few, so none is taken as heavy; 39: at most the call's rows minus one.
# The last three: a shared expert of its own bit width or size, so launches of its own beside the split.
@pytest.mark.parametrize("bits,meta,out,limit,shared", [
    (4, BF16, fmt.OUT_FP16, 8, ()), (8, BF16, fmt.OUT_FP32, 8, ()), (8, FP16, fmt.OUT_FP16, 9, ()), (4, BF16, fmt.OUT_FP32, 16, ()),
    (4, FP16, fmt.OUT_FP16, 39, ()), (4, BF16, fmt.OUT_FP16, 8, (256, 8)), (8, FP16, fmt.OUT_FP32, 9, (256, 4)),
    (4, BF16, fmt.OUT_FP32, 8, (512, 4))])
@pytest.mark.parametrize("entry", ["decode", "prefill"])
def test_calls_split_between_the_two_kernels_match_the_oracle(bits, meta, out, limit, shared, entry, monkeypatch):
    monkeypatch.setenv("NVMAI_CUDA_STREAM_ROWS", str(limit))
    d, f, tokens = 512, 256, 40
    host = _host_layer(811 + limit, bits, meta, d, f, 32, *shared)
    cfg = MoEConfig(d=d, f=f, shared_f=host["shared"][0][0].shape[0], num_experts=32, top_k=8, routed_bits=bits,
                    shared_bits=shared[1] if shared else bits, meta_dtype=meta, out_dtype=out, max_tokens=tokens)
    assert _worst_error(host, cfg, entry, tokens, range(0, tokens, 3)) < _tol(meta, out, entry)


# The split a call takes by itself at the benchmark's shape (256 experts, 8-bit codes), evenly routed: streamed below 6 rows
# per expert, experts above 16 rows on the tcgen05 kernel between 6 and 24 (two passes a code), all of them above; the
# rows of the first, a middle and the last token.
@pytest.mark.parametrize("tokens", [190, 200, 760, 780])
def test_default_split_matches_the_oracle(tokens):
    host = _host_layer(90, 8, BF16, 2048, 512, 256)
    cfg = MoEConfig(d=2048, f=512, shared_f=512, num_experts=256, top_k=8, routed_bits=8, shared_bits=8, meta_dtype=BF16,
                    out_dtype=fmt.OUT_FP32, max_tokens=tokens)
    assert _worst_error(host, cfg, "prefill", tokens, (0, tokens // 2, tokens - 1)) < _tol(BF16, fmt.OUT_FP32, "prefill")


# A stack of several rows: 3 rows the staged kernels, 4 and more the batched experts' with the norm of the next layer's
# rows in the reduction; 2304: a row longer than that norm takes, 8: the most rows the route log keeps.  Layer by layer with
# rms_renorm, whose reduction tree is the same, the result is the same bit for bit.
@pytest.mark.parametrize("rows,bits,out,d,f,experts", [(3, 4, fmt.OUT_FP32, 512, 256, 64), (4, 8, fmt.OUT_FP32, 256, 128, 128),
                                                       (8, 4, fmt.OUT_FP16, 2048, 512, 256), (9, 4, fmt.OUT_FP32, 2304, 128, 32)])
def test_stack_of_rows_equals_its_layers_one_by_one(rows, bits, out, d, f, experts):
    layers = 3
    torch = gu.torch_cuda()
    cfg = MoEConfig(d=d, f=f, shared_f=f, num_experts=experts, top_k=8, routed_bits=bits, shared_bits=bits, meta_dtype=BF16,
                    out_dtype=out, max_tokens=rows, num_layers=layers)
    moe = MoE(cfg)
    keep = [synthetic.device_layer(90 + 3 * l + bits, d=d, f=f, shared_f=f, num_experts=experts, routed_bits=bits, shared_bits=bits,
                                   meta=BF16) for l in range(layers)]
    for l, dev in enumerate(keep):
        synthetic.register_device_layer(moe, l, dev)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        x0 = torch.randn((rows, d), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)).half()
        kind = torch.float16 if out == fmt.OUT_FP16 else torch.float32
        y, again, y1 = (torch.zeros((rows, d), dtype=kind, device="cuda") for _ in range(3))
        idx = torch.empty((rows, 8), dtype=torch.int32, device="cuda")
        x_next = torch.empty((rows, d), dtype=torch.float16, device="cuda")
        moe.stack_decode(x0, rows, y, stream=st)
        moe.stack_decode(x0, rows, again, stream=st)
        moe.synchronize(st)
        log = moe.read_route_log_rows(rows) if rows <= 8 else None
        x = x0
        for l in range(layers):
            moe.layer_decode(l, x, rows, h2_out=y1, out_idx=idx, stream=st)
            moe.rms_renorm(y1, rows, x_next, stream=st)
            moe.synchronize(st)
            if log is not None:
                np.testing.assert_array_equal(log[l].astype(np.int64), idx.cpu().numpy())
            x = x_next.clone()
    assert torch.equal(y, again) and bool(torch.isfinite(y).all())
    assert torch.equal(y, y1)


# 8 experts see every row, 27 units of gate/up: 62 rows, items of 96, two sets of accumulators and two A slots; 90 rows, items of
# 128, one set that all warps empty and four slots; 150 rows, items of 176, one set, two slots.
@pytest.mark.parametrize("bits,meta,out,tokens", [(4, BF16, fmt.OUT_FP16, 62), (8, FP16, fmt.OUT_FP32, 62), (4, BF16, fmt.OUT_FP32, 90),
                                                  (8, FP16, fmt.OUT_FP16, 90), (4, FP16, fmt.OUT_FP16, 150), (8, BF16, fmt.OUT_FP16, 150)])
@pytest.mark.parametrize("entry", ["decode", "prefill"])
def test_items_of_every_tensor_memory_plan_match_the_oracle(bits, meta, out, tokens, entry, monkeypatch):
    monkeypatch.setenv("NVMAI_CUDA_STREAM_ROWS", "0")
    host = _host_layer(900 + tokens, bits, meta, 768, 384, 8)
    cfg = MoEConfig(d=768, f=384, shared_f=384, num_experts=8, top_k=8, routed_bits=bits, shared_bits=bits, meta_dtype=meta,
                    out_dtype=out, max_tokens=tokens)
    assert _worst_error(host, cfg, entry, tokens, sorted({0, 31, tokens // 2, tokens - 1})) < _tol(meta, out, entry)


# Every plan by name, with more units than SMs, so that slots and parities go on from unit to unit, odd numbers of slots and of
# stages among them (d = 768: 13 stages of a 4-bit unit, 25 of an 8-bit one).  plan: rows of the longest item, sets of accumulators,
# A slots.  8192 / 384: the ring of rows leaves items of 80.
@pytest.mark.parametrize("bits,out,tokens,d,f,experts,plan", [
    (4, fmt.OUT_FP16, 64, 768, 384, 64, (48, 2, 5)), (8, fmt.OUT_FP32, 64, 768, 384, 64, (48, 2, 5)),
    (4, fmt.OUT_FP32, 300, 768, 640, 64, (96, 2, 2)), (8, fmt.OUT_FP16, 300, 768, 640, 64, (96, 2, 2)),
    (4, fmt.OUT_FP16, 300, 768, 768, 32, (128, 1, 4)), (8, fmt.OUT_FP32, 300, 768, 768, 32, (128, 1, 4)),
    (4, fmt.OUT_FP32, 512, 768, 768, 32, (160, 1, 3)), (8, fmt.OUT_FP16, 512, 768, 768, 32, (160, 1, 3)),
    (4, fmt.OUT_FP16, 640, 768, 768, 32, (192, 1, 2)),
    (4, fmt.OUT_FP32, 300, 8192, 384, 64, (80, 2, 3)),
])
def test_units_walk_through_every_tensor_memory_plan(bits, out, tokens, d, f, experts, plan, monkeypatch):
    monkeypatch.setenv("NVMAI_CUDA_STREAM_ROWS", "0")
    cfg = MoEConfig(d=d, f=f, shared_f=f, num_experts=experts, top_k=8, routed_bits=bits, shared_bits=bits, meta_dtype=BF16,
                    out_dtype=out, max_tokens=tokens)
    assert MoE(cfg).debug_item_plan(tokens, 0) == plan
    host = _host_layer(950 + tokens, bits, BF16, d, f, experts)
    assert _worst_error(host, cfg, "prefill", tokens, sorted({0, 31, tokens // 2, tokens - 1})) < _tol(BF16, out, "prefill")


# Routing in blocks of 8 tokens (up to 1024) and of 32, with a last block of one; the reduction walks more rows than its grid.
@pytest.mark.parametrize("tokens", [33, 1024, 1025, 1409])
def test_rows_at_the_borders_of_the_routing_blocks_match_the_oracle(tokens):
    host = _host_layer(77, 4, BF16, 256, 128, 256)
    cfg = MoEConfig(d=256, f=128, shared_f=128, num_experts=256, top_k=8, routed_bits=4, shared_bits=4, meta_dtype=BF16,
                    out_dtype=fmt.OUT_FP32, max_tokens=tokens)
    sample = sorted({t for t in (0, 7, 8, 31, 32, 443, 444, 445, 1023, 1024, tokens - 1) if t < tokens})
    assert _worst_error(host, cfg, "prefill", tokens, sample) < _tol(BF16, fmt.OUT_FP32, "prefill")


# More than 128 routing blocks of 32 tokens: a block's first pair is found from the counts of its own segment of 128 blocks and the
# totals of those in front (8225: three segments, the last of two blocks).  Up to 768 rows the kernels know of one segment only.
@pytest.mark.parametrize("tokens", [768, 769, 4096, 4097, 8225])
def test_rows_past_a_segment_of_routing_blocks_match_the_oracle(tokens):
    host = _host_layer(78, 4, BF16, 256, 128, 256)
    cfg = MoEConfig(d=256, f=128, shared_f=128, num_experts=256, top_k=8, routed_bits=4, shared_bits=4, meta_dtype=BF16,
                    out_dtype=fmt.OUT_FP32, max_tokens=tokens)
    sample = sorted({t for t in (0, 759, 760, 767, 4063, 4064, 4095, 4096, 8191, 8192, 8223, tokens - 1) if t < tokens})
    assert _worst_error(host, cfg, "prefill", tokens, sample) < _tol(BF16, fmt.OUT_FP32, "prefill")


# A caller's routing may name one expert eight times in every row: 256 pairs of a block on one expert.  The row's share is then
# that expert's output, eight eighths of it (fp32 additions: 8 x 2^-24).
@pytest.mark.parametrize("tokens", [40, 1100])
def test_an_expert_named_by_every_slot_of_every_row(tokens):
    torch = gu.torch_cuda()
    cfg = MoEConfig(d=256, f=128, shared_f=0, shared_gate_kind=fmt.GATE_NONE, num_experts=16, top_k=8, routed_bits=4, shared_bits=4,
                    meta_dtype=BF16, out_dtype=fmt.OUT_FP32, max_tokens=tokens)
    moe = MoE(cfg)
    dev = synthetic.device_layer(5, d=256, f=128, shared_f=0, num_experts=16, routed_bits=4, shared_bits=4, meta=BF16)
    synthetic.register_device_layer(moe, 0, dev)
    x = torch.randn((tokens, 256), device="cuda", generator=torch.Generator(device="cuda").manual_seed(9)).half()
    same = torch.full((tokens, 8), 3, dtype=torch.int32, device="cuda")
    once = torch.arange(8, dtype=torch.int32, device="cuda").repeat(tokens, 1)
    share, want = (torch.zeros((tokens, 256), device="cuda") for _ in range(2))
    moe.routed_partial(0, x, tokens, same, torch.full((tokens, 8), 0.125, dtype=torch.float16, device="cuda"), share)
    moe.routed_partial(0, x, tokens, once, (once == 3).half(), want)
    moe.synchronize()
    assert bool(torch.isfinite(want).all()) and float(want.abs().max()) > 0
    assert float((share - want).norm() / want.norm()) < 2e-6
