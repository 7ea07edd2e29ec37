"""A row of a decode batch has the bits of a call of its own, on the kernels that a call takes by default."""
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
for p_ in (ROOT, ROOT / "tests"):
    if str(p_) not in sys.path:
        sys.path.insert(0, str(p_))

pytestmark = pytest.mark.gpu

from nvmai_b200 import MoE, MoEConfig, synthetic      # noqa: E402
from nvmai_b200 import format as fmt                  # noqa: E402
import gpu_util as gu                                 # noqa: E402

BF16, FP16 = fmt.META_BF16, fmt.META_FP16
DENSE, AFF8 = fmt.ROUTER_DENSE_F16, fmt.ROUTER_AFFINE8


def _layer(seed, cfg):
    """zero-mean weights on the device; affine router and gate rows where the configuration asks for them"""
    torch = gu.torch_cuda()
    dev = synthetic.device_layer(seed, d=cfg.d, f=cfg.f, shared_f=cfg.shared_f, num_experts=cfg.num_experts,
                                 routed_bits=cfg.routed_bits, shared_bits=cfg.shared_bits, meta=cfg.meta_dtype)
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    if cfg.router_kind != DENSE:
        dev["router"] = synthetic._device_affine(torch, gen, cfg.num_experts, cfg.d, cfg.router_kind, cfg.meta_dtype, "cuda")
    if cfg.shared_f and cfg.shared_gate_kind not in (DENSE, fmt.GATE_NONE):
        dev["gate"] = synthetic._device_affine(torch, gen, 1, cfg.d, cfg.shared_gate_kind, cfg.meta_dtype, "cuda")
    return dev


def _config(bits, meta, out, rows, d, f, experts, router, **other):
    kw = dict(d=d, f=f, shared_f=f, num_experts=experts, top_k=8, routed_bits=bits, shared_bits=bits, router_kind=router,
              shared_gate_kind=router, meta_dtype=meta, out_dtype=out, max_tokens=rows)
    kw.update(other)
    return MoEConfig(**kw)


def _check_rows_alone(cfg, rows, seed):
    torch = gu.torch_cuda()
    moe = MoE(cfg)
    dev = _layer(seed, cfg)
    synthetic.register_device_layer(moe, 0, dev)
    x = torch.randn((rows, cfg.d), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).half()
    kind = torch.float16 if cfg.out_dtype == fmt.OUT_FP16 else torch.float32

    def call(first, n):
        h2 = torch.zeros((n, cfg.d), dtype=kind, device="cuda")
        hidden = torch.full((n, cfg.d), 0.75, dtype=kind, device="cuda")
        idx = torch.zeros((n, 8), dtype=torch.int32, device="cuda")
        w = torch.zeros((n, 8), dtype=torch.float16, device="cuda")
        moe.layer_decode(0, x[first:first + n], n, hidden=hidden, h2_out=h2, out_idx=idx, out_w=w)
        moe.synchronize()
        return idx, w, h2, hidden

    batch = call(0, rows)
    assert bool(torch.isfinite(batch[2]).all())
    for t in range(rows):
        for name, all_rows, one in zip(("idx", "w", "h2", "hidden"), batch, call(t, 1)):
            assert torch.equal(all_rows[t], one[0]), f"row {t}: {name}"


# Rows of 4096 values: parts of two quads of groups in both phases of the streaming kernel; 1536: three quads in the down
# projection.
@pytest.mark.parametrize("bits,meta,out,rows,d,f", [
    (4, BF16, fmt.OUT_FP16, 5, 4096, 1024), (8, BF16, fmt.OUT_FP32, 4, 4096, 1024), (8, FP16, fmt.OUT_FP16, 9, 4096, 512),
    (4, BF16, fmt.OUT_FP32, 13, 2048, 1536), (4, FP16, fmt.OUT_FP32, 6, 2048, 1024)])
def test_long_rows_equal_calls_of_their_own(bits, meta, out, rows, d, f):
    cfg = _config(bits, meta, out, rows, d, f, 32, AFF8)
    _check_rows_alone(cfg, rows, seed=100 + rows)


# Affine routers (what a repacked artifact has): the routing kernel selects from the logits of the rows' blocks.  4 rows: a
# block's rows are spread over four; 9: an odd number a block; 31: the most rows.  1: no batched kernels at all.
@pytest.mark.parametrize("bits,meta,out,rows,router", [
    (4, BF16, fmt.OUT_FP16, 1, AFF8), (4, BF16, fmt.OUT_FP16, 4, AFF8), (8, FP16, fmt.OUT_FP32, 9, fmt.ROUTER_AFFINE4),
    (4, FP16, fmt.OUT_FP16, 31, AFF8)])
def test_rows_of_an_affine_router_equal_calls_of_their_own(bits, meta, out, rows, router):
    cfg = _config(bits, meta, out, rows, 512, 256, 256, router)
    _check_rows_alone(cfg, rows, seed=200 + rows)


# Dense routers: up to 31 rows the single-row router's order of additions and the streaming kernel, also where few experts
# hold the rows (8 experts: 31 rows each); a shape of the streaming kernel's (2048 / 512) and others; no shared expert; a
# shared expert of its own bit width.
@pytest.mark.parametrize("bits,meta,out,rows,d,f,experts,other", [
    (4, BF16, fmt.OUT_FP32, 4, 2048, 512, 256, {}), (8, BF16, fmt.OUT_FP16, 9, 2048, 512, 64, {}),
    (4, FP16, fmt.OUT_FP16, 31, 2048, 512, 256, {}), (4, BF16, fmt.OUT_FP32, 31, 512, 128, 8, {}),
    (8, FP16, fmt.OUT_FP32, 13, 768, 384, 128, {}), (4, BF16, fmt.OUT_FP16, 7, 256, 128, 128, {"shared_f": 0}),
    (4, BF16, fmt.OUT_FP32, 11, 512, 256, 128, {"shared_bits": 8, "shared_f": 128}), (4, BF16, fmt.OUT_FP16, 20, 4096, 512, 16, {})])
def test_rows_of_a_dense_router_equal_calls_of_their_own(bits, meta, out, rows, d, f, experts, other):
    cfg = _config(bits, meta, out, rows, d, f, experts, DENSE, **other)
    _check_rows_alone(cfg, rows, seed=300 + rows)


# From 32 rows on the dense router is a GEMM whose K is split over four, two or one block by the number of rows (at 256
# experts on 148 SMs up to 1152, 2368 and more rows; at 128 experts up to 2368, 4736 and more): the logits, and so the
# routing, are the same for any number.
@pytest.mark.parametrize("d,experts,some,most", [(256, 256, (40, 1100, 1500, 2368), 2500), (1280, 256, (40, 1152, 1500), 2500),
                                                 (256, 128, (40, 2368, 2369, 4736), 4800)])
def test_routing_of_a_row_does_not_depend_on_the_rows_beside_it(d, experts, some, most):
    torch = gu.torch_cuda()
    cfg = _config(4, BF16, fmt.OUT_FP16, most, d, 128, experts, DENSE)
    moe = MoE(cfg)
    dev = _layer(17, cfg)
    synthetic.register_device_layer(moe, 0, dev)
    x = torch.randn((most, d), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5)).half()

    def routing(rows):
        idx = torch.zeros((rows, 8), dtype=torch.int32, device="cuda")
        w = torch.zeros((rows, 8), dtype=torch.float16, device="cuda")
        y = torch.zeros((rows, d), dtype=torch.float16, device="cuda")
        moe.layer_prefill(0, x, rows, y_out=y, out_idx=idx, out_w=w)
        moe.synchronize()
        return idx, w

    idx, w = routing(most)
    for rows in some:
        some_idx, some_w = routing(rows)
        assert torch.equal(some_idx, idx[:rows]) and torch.equal(some_w, w[:rows]), rows


# A stack of rows on buffers it has not seen: the graph belongs to the row count, not to the buffers, and the caller's rows
# are read and written.  2: the staged kernels, 5: the batched ones.
@pytest.mark.parametrize("rows", [2, 5])
def test_stack_graphs_are_not_kept_by_buffer(rows):
    torch = gu.torch_cuda()
    cfg = _config(4, BF16, fmt.OUT_FP32, 40, 256, 128, 128, DENSE, num_layers=9)
    moe = MoE(cfg)
    keep = [_layer(31 + l, cfg) for l in range(9)]
    for l, dev in enumerate(keep):
        synthetic.register_device_layer(moe, l, dev)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        x = torch.randn((6, rows, cfg.d), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)).half()
        y = torch.zeros((6, rows, cfg.d), device="cuda")
        for i in range(6):
            moe.stack_decode(x[i], rows, y[i], stream=st)
        again = torch.zeros_like(y)
        for i in (3, 0, 5, 1, 4, 2):
            moe.stack_decode(x[i], rows, again[i], stream=st)
        moe.synchronize(st)
    plain = torch.zeros_like(y)
    torch.cuda.synchronize()
    for i in range(6):                                    # the default stream: plain launches, the caller's buffers
        moe.stack_decode(x[i], rows, plain[i], stream=0)
    moe.synchronize()
    assert moe.debug_stack_graphs() == 1
    assert torch.equal(y, again) and torch.equal(y, plain) and bool((y != 0).any())


def test_stack_graphs_are_bounded():
    torch = gu.torch_cuda()
    cfg = _config(4, BF16, fmt.OUT_FP32, 40, 256, 128, 128, DENSE, num_layers=8)
    moe = MoE(cfg)
    keep = [_layer(41 + l, cfg) for l in range(8)]
    for l, dev in enumerate(keep):
        synthetic.register_device_layer(moe, l, dev)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        x = torch.randn((40, cfg.d), device="cuda").half()
        y = torch.zeros((40, cfg.d), device="cuda")
        for rows in range(2, 41):                         # the last of them as plain launches
            moe.stack_decode(x, rows, y, stream=st)
        moe.synchronize(st)
    plain = torch.zeros_like(y)
    torch.cuda.synchronize()
    moe.stack_decode(x, 40, plain, stream=0)
    moe.synchronize()
    assert moe.debug_stack_graphs() == 32
    assert torch.equal(y, plain)


# A handle that holds a part of the experts (set_expert_map): the whole-block calls leave the others out, as if their
# weights were zero, on every path: 1 row, a few, grouped, a stack; top-2 without a shared expert: the stages that read the
# indices instead of selecting.
@pytest.mark.parametrize("rows,other", [(1, {}), (3, {}), (6, {}), (30, {}), (3, {"top_k": 2, "shared_f": 0})])
@pytest.mark.parametrize("entry", ["layer", "stack"])
def test_calls_on_a_part_of_the_experts_leave_the_others_out(rows, other, entry):
    torch = gu.torch_cuda()
    cfg = _config(4, BF16, fmt.OUT_FP32, 32, 256, 128, 64, DENSE, **other)
    dev = _layer(53, cfg)
    held = [e for e in range(64) if e % 3 != 1]
    gone = [e for e in range(64) if e % 3 == 1]
    part = dict(dev, experts=dev["experts"][held].clone())
    off, meta_bytes = dev["offsets"], 128 * (256 // 64) * 2
    for name in ("gate_s", "gate_b", "up_s", "up_b", "down_s", "down_b"):      # (all six are as long: 256 x 128 / 64)
        dev["experts"][gone, off[name]:off[name] + meta_bytes] = 0
    x = torch.randn((rows, cfg.d), device="cuda", generator=torch.Generator(device="cuda").manual_seed(rows)).half()

    def run(weights, expert_map):
        moe = MoE(cfg)
        if expert_map is not None:
            moe.set_expert_map(expert_map)
        synthetic.register_device_layer(moe, 0, weights)
        y = torch.zeros((rows, cfg.d), device="cuda")
        if entry == "layer":
            moe.layer_decode(0, x, rows, h2_out=y)
        else:
            moe.stack_decode(x, rows, y)
        moe.synchronize()
        return y

    want = run(dev, None)
    got = run(part, [held.index(e) if e in held else 0xFFFFFFFF for e in range(64)])
    assert bool(torch.isfinite(want).all()) and bool((want != 0).any())
    assert torch.equal(got, want) or float((got - want).norm() / want.norm()) < 1e-6
