"""Stage 3 of a decode call polls the activations as tagged words; under capture it waits for stage 2 and reads plain arrays.
Both give the same bits, over the rows and row lengths that the words are made for and past them."""
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

F16, F32 = fmt.OUT_FP16, fmt.OUT_FP32


@pytest.mark.parametrize("rows,d,f,shared_f,bits,out", [
    (1, 2048, 512, 512, 4, F16), (1, 2048, 512, 512, 4, F32),       # one wave of each stage
    (2, 2048, 512, 512, 8, F16), (3, 2048, 512, 512, 8, F32),       # more blocks than fit at once
    (3, 256, 128, 128, 4, F16), (3, 256, 64, 192, 8, F32),          # the shortest rows; expert and shared rows of two lengths
    (2, 1024, 1024, 320, 4, F16),                                   # the longest row of halves, a ragged last step
    (2, 512, 576, 512, 4, F32),                                     # longer than the words of wide rows: none
    (1, 512, 448, 0, 4, F32),                                       # no shared expert, two steps a half of a row
])
def test_handed_over_rows_have_the_bits_of_plain_ones(rows, d, f, shared_f, bits, out):
    torch = gu.torch_cuda()
    cfg = MoEConfig(d=d, f=f, shared_f=shared_f, num_experts=64, top_k=8, routed_bits=bits, shared_bits=bits,
                    shared_gate_kind=fmt.ROUTER_DENSE_F16 if shared_f else fmt.GATE_NONE, out_dtype=out, max_tokens=rows)
    moe = MoE(cfg)
    dev = synthetic.device_layer(7 * d + f, d=d, f=f, shared_f=shared_f, num_experts=64, routed_bits=bits, shared_bits=bits)
    synthetic.register_device_layer(moe, 0, dev)
    gen = torch.Generator(device="cuda").manual_seed(d + rows)
    kind = torch.float16 if out == F16 else torch.float32
    start = (torch.randn((rows, d), device="cuda", generator=gen) * 4).to(kind)
    delta = torch.randn((rows, d), device="cuda", generator=gen).half()
    norm, next_norm = ((torch.rand(d, device="cuda", generator=gen) + 0.5).to(torch.bfloat16) for _ in range(2))
    hidden = start.clone()
    got = [torch.empty((rows, d), dtype=torch.float16, device="cuda"), torch.empty((rows, d), dtype=kind, device="cuda"),
           torch.empty((rows, 8), dtype=torch.int32, device="cuda"), torch.empty((rows, 8), dtype=torch.float16, device="cuda")]

    def call(n, stream):
        hidden.copy_(start)
        moe.layer_decode_fused_norms(0, hidden, norm, 1e-6, n, next_norm, 1e-5, got[0], attn_delta=delta, h2_out=got[1],
                                     out_idx=got[2], out_w=got[3], stream=stream)

    def result(n):
        moe.synchronize()
        torch.cuda.synchronize()
        return [t[:n].clone() for t in (hidden, *got)]

    call(rows, torch.cuda.current_stream())
    first = result(rows)
    assert all(bool(torch.isfinite(t.float()).all()) for t in first)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(rows, torch.cuda.current_stream())
    for _ in range(2):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(first, result(rows)))
    for n in (1, rows, 1, rows) * 10:          # words of an earlier call, of more rows or fewer, lie in the way
        call(n, torch.cuda.current_stream())
        assert all(torch.equal(a[:n], b) for a, b in zip(first, result(n)))


def _block(torch, rows, out, seed, next_norm=True):
    """A handle with one polling layer and a decode call of it; -> (moe, call(stream), outputs)."""
    d, f = 512, 256
    cfg = MoEConfig(d=d, f=f, shared_f=f, num_experts=64, top_k=8, routed_bits=4, shared_bits=4,
                    shared_gate_kind=fmt.ROUTER_DENSE_F16, out_dtype=out, max_tokens=3)
    moe = MoE(cfg)
    dev = synthetic.device_layer(seed, d=d, f=f, shared_f=f, num_experts=64, routed_bits=4, shared_bits=4)
    synthetic.register_device_layer(moe, 0, dev)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = torch.float16 if out == F16 else torch.float32
    start = (torch.randn((rows, d), device="cuda", generator=gen) * 4).to(kind)
    norm = (torch.rand(d, device="cuda", generator=gen) + 0.5).to(torch.bfloat16)
    hidden, x_next = start.clone(), torch.zeros((rows, d), dtype=torch.float16, device="cuda")

    def call(stream):
        hidden.copy_(start)
        if next_norm:
            moe.layer_decode_fused_norms(0, hidden, norm, 1e-6, rows, norm, 1e-6, x_next, stream=stream)
        else:
            moe.layer_decode_prenorm(0, hidden, norm, 1e-6, rows, stream=stream)

    return moe, call, (hidden, x_next), dev


# The polls of stage 3 (halves, fp32 values, the block of the next norm) run out, from the host side: stage 3 waits for words that
# nobody writes.  Waits are cut to 20 ms; the call ends, the time-out is reported once, and the next call has the bits of the first.
@pytest.mark.parametrize("rows,out,next_norm", [(1, F16, True), (3, F32, True), (2, F16, False)])
def test_a_hand_over_that_never_comes_times_out_and_the_next_call_runs(rows, out, next_norm):
    from nvmai_b200 import _lib
    from nvmai_b200.moe import debug_set_wait_limit
    torch = gu.torch_cuda()
    moe, call, outs, _keep = _block(torch, rows, out, 31 + rows, next_norm)
    st = torch.cuda.current_stream()
    call(st)
    moe.synchronize()
    good = [t.clone() for t in outs]
    debug_set_wait_limit(20_000_000)
    try:
        moe.debug_drop_handover()
        call(st)
        with pytest.raises(_lib.NvmaiError) as err:
            moe.synchronize()
        assert err.value.code == _lib.ETIMEOUT
    finally:
        debug_set_wait_limit(0)
    for _ in range(2):
        call(st)
        moe.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(good, outs))


def test_two_handles_poll_on_two_streams_at_once():
    torch = gu.torch_cuda()
    made = [_block(torch, rows, out, 50 + rows) for rows, out in ((1, F16), (3, F32))]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in made]
    good = []
    for (moe, call, outs, _keep), st in zip(made, streams):
        with torch.cuda.stream(st):
            call(st)
        moe.synchronize(st)
        good.append([t.clone() for t in outs])
    torch.cuda.synchronize()
    for _ in range(50):
        for (moe, call, outs, _keep), st in zip(made, streams):
            with torch.cuda.stream(st):
                call(st)
    for (moe, call, outs, _keep), st, want in zip(made, streams, good):
        moe.synchronize(st)
        assert all(torch.equal(a, b) for a, b in zip(want, outs))
