// Launchers of the batched path: see batch_path.h.
#include "batch_path.h"

#include <algorithm>
#include <type_traits>

#include "batch_rows.cuh"
#include "expert_gemm.cuh"
#include "launch.h"
#include "stream_gemm.cuh"

namespace nvmai {

namespace {
constexpr size_t kMaxBlockSmem = 227 * 1024;
}

EgPlan eg_plan(EgParams &p, int phase, uint32_t want_cap) {
    const uint32_t n_main = p.kdim / 64, n_kb = n_main + bp_extra_cols(p.kdim, phase == 0 ? 1 : 2) / 64;
    const size_t fixed = 2048 + (size_t)kEgChunks * kEgChunkBytes;           // alignment slack, barriers, code ring
    p.meta_slot_bytes = 128 * n_main * 4;
    p.meta_slots = (size_t)4 * p.meta_slot_bytes <= 64 * 1024 ? 4 : 2;
    auto meta_ring = [&]() { return ((size_t)p.meta_slots * p.meta_slot_bytes + 1023) & ~(size_t)1023; };
    size_t meta = meta_ring();
    if (fixed + meta + 2 * 2048 > kMaxBlockSmem) return EgPlan{0, 0};
    size_t avail = kMaxBlockSmem - fixed - meta;
    uint32_t cap = (want_cap + 15) / 16 * 16;
    if (phase == 0) {
        // three K blocks of rows in flight at least
        cap = std::min({cap, 192u, (uint32_t)(avail / 3 / 128) / 16 * 16});
        p.resident = 0;
    } else {
        cap = std::min(cap, 128u);
        const uint32_t fits = (uint32_t)(avail / (n_kb * 128)) / 16 * 16;    // rows whose every K block stays
        p.resident = n_kb <= kEgMaxRowSlots && (fits >= cap || fits >= 48) ? 1 : 0;
        cap = std::min(cap, p.resident ? fits : (uint32_t)(avail / 3 / 128) / 16 * 16);
    }
    if (cap == 0) return EgPlan{0, 0};
    p.acc_tile_off = phase == 0 ? cap : 0;
    p.acc_stride = phase == 0 ? 2 * cap : cap;
    // two sets of accumulators where at least two A slots remain beside them; what is left goes to the A slots
    p.acc_slots = 2 * p.acc_stride + 2 * kEgSlotCols <= kEgCols ? 2 : 1;
    p.a_slots = std::min(kEgMaxPairs, (kEgCols - p.acc_slots * p.acc_stride) / kEgSlotCols);
    p.a_col = kEgCols - p.a_slots * kEgSlotCols;
    p.acc_slots = std::min(kEgMaxAcc, p.a_col / p.acc_stride);
    if (phase == 0 && p.acc_slots == 1) {       // the scales of the next unit come while the accumulators are emptied
        p.meta_slots = 2;
        meta = meta_ring();
        avail = kMaxBlockSmem - fixed - meta;
    }
    p.row_slot_bytes = cap * 128;
    p.row_slots = (uint32_t)std::min<size_t>(kEgMaxRowSlots, avail / p.row_slot_bytes);
    p.row_ring_off = (uint32_t)(1024 + (size_t)kEgChunks * kEgChunkBytes + meta);
    p.cap = cap;
    return EgPlan{cap, fixed + meta + (size_t)p.row_slots * p.row_slot_bytes};
}

cudaError_t eg_launch(int phase, uint32_t bits, uint32_t meta, uint32_t out_dtype, bool split, const EgArgs &args, uint32_t blocks,
                      size_t smem, cudaStream_t st) {
    auto go = [&](auto B, auto M, auto O, auto P, auto S) {
        return launch_pdl(expert_gemm_kernel<decltype(B)::value, decltype(M)::value, decltype(O)::value, decltype(P)::value,
                                             decltype(S)::value>, dim3(blocks), dim3(kEgThreads), smem, st, true, args);
    };
    using std::integral_constant;
    auto with_split = [&](auto B, auto O, auto P) {
        if (meta == META_BF16) return go(B, integral_constant<int, META_BF16>{}, O, P, integral_constant<bool, false>{});
        if (split) return go(B, integral_constant<int, META_FP16>{}, O, P, integral_constant<bool, true>{});
        return go(B, integral_constant<int, META_FP16>{}, O, P, integral_constant<bool, false>{});
    };
    auto with_out = [&](auto B) {      // phase 1 does not depend on the activations' type
        if (phase == 1) return with_split(B, integral_constant<int, OUT_F32>{}, integral_constant<int, 1>{});
        if (out_dtype == OUT_F16) return with_split(B, integral_constant<int, OUT_F16>{}, integral_constant<int, 0>{});
        return with_split(B, integral_constant<int, OUT_F32>{}, integral_constant<int, 0>{});
    };
    if (bits == 4) return with_out(integral_constant<int, 4>{});
    return with_out(integral_constant<int, 8>{});
}

// Are the parts of a row (an eighth of its groups in gate/up, a half in down) one quad of groups each (1), several whole
// quads (2) or neither (0)?  At 4096 inputs the unit of 128 features that 0 takes leaves no room for its scales: 5 rows of
// 4096 / 1024, 8-bit, took 307 us through the tcgen05 kernel and 252 as separate rows; in units of 64 features 142.
static int sg_quads(int phase, uint32_t kdim) {
    const uint32_t part = kdim / 64 / (phase == 0 ? 8 : 2);
    return kdim / 64 % (phase == 0 ? 32 : 8) != 0 ? 0 : part == 4 ? 1 : 2;
}

size_t sg_plan(SgParams &p, int phase, uint32_t nb, bool wide) {
    const uint32_t groups = p.kdim / 64, cols = 8 * nb;
    const uint32_t rows = phase == 1 ? 256 : sg_quads(0, p.kdim) != 0 ? 64 : 128;        // features or down rows of a unit
    if (p.out_cols % rows != 0) return 0;
    p.units_per_item = p.out_cols / rows;
    p.cap = cols;
    p.meta_bytes = rows * groups * 2 * (phase == 0 ? 4 : 2);
    auto up = [](size_t v) { return (v + 127) & ~(size_t)127; };
    size_t fixed = 2 * p.meta_bytes + up((size_t)cols * (p.kdim * 2 + 16)) + (phase == 1 && wide ? up((size_t)cols * p.kdim * 4) : 0) +
                   up((size_t)cols * (groups + 4) * 4) + up(cols * 4 + (phase == 0 ? 2 * 8 * 4 * nb * 32 * 4 : 0));
    if (fixed + 2048 + 2 * kSgStageBytes > kMaxBlockSmem) return 0;
    p.stages = (uint32_t)std::min<size_t>(kSgMaxStages, (kMaxBlockSmem - 2048 - fixed) / kSgStageBytes);
    size_t o = 1024 + (size_t)p.stages * kSgStageBytes;
    p.meta_off = (uint32_t)o; o += 2 * p.meta_bytes;
    p.x_off = (uint32_t)o; o += up((size_t)cols * (p.kdim * 2 + 16));
    p.raw_off = (uint32_t)o; o += phase == 1 && wide ? up((size_t)cols * p.kdim * 4) : 0;
    p.sum_off = (uint32_t)o; o += up((size_t)cols * (groups + 4) * 4);
    p.scale_off = (uint32_t)o; o += up(cols * 4 + (phase == 0 ? 2 * 8 * 4 * nb * 32 * 4 : 0));
    return o + 1024;
}

cudaError_t sg_launch(int phase, uint32_t bits, uint32_t meta, uint32_t out_dtype, uint32_t nb, const SgArgs &args, uint32_t blocks,
                      size_t smem, cudaStream_t st) {
    using std::integral_constant;
    const int quads = sg_quads(phase, args.p.kdim);
    auto go = [&](auto B, auto M, auto O, auto P, auto N, auto F) {
        return launch_pdl(stream_gemm_kernel<decltype(B)::value, decltype(M)::value, decltype(O)::value, decltype(P)::value, decltype(N)::value,
                                             decltype(F)::value>, dim3(blocks), dim3(kSgThreads + 32), smem, st, true, args);
    };
    auto with_quads = [&](auto B, auto M, auto O, auto P, auto N) {
        if (quads == 0) return go(B, M, O, P, N, integral_constant<int, 0>{});
        if (quads == 1) return go(B, M, O, P, N, integral_constant<int, 1>{});
        if constexpr (decltype(P)::value == 0 && decltype(N)::value == 2) return cudaErrorInvalidValue;   // no room for 16 rows (sg_plan)
        else return go(B, M, O, P, N, integral_constant<int, 2>{});
    };
    auto with_n = [&](auto B, auto M, auto O, auto P) {
        if (nb == 1) return with_quads(B, M, O, P, integral_constant<int, 1>{});
        return with_quads(B, M, O, P, integral_constant<int, 2>{});
    };
    auto with_p = [&](auto B, auto M, auto O) {
        if (phase == 0) return with_n(B, M, O, integral_constant<int, 0>{});
        return with_n(B, M, O, integral_constant<int, 1>{});
    };
    auto with_o = [&](auto B, auto M) {
        if (out_dtype == OUT_F16) return with_p(B, M, integral_constant<int, OUT_F16>{});
        return with_p(B, M, integral_constant<int, OUT_F32>{});
    };
    auto with_m = [&](auto B) {
        if (meta == META_BF16) return with_o(B, integral_constant<int, META_BF16>{});
        return with_o(B, integral_constant<int, META_FP16>{});
    };
    if (bits == 4) return with_m(integral_constant<int, 4>{});
    return with_m(integral_constant<int, 8>{});
}

cudaError_t bp_pack_x(const PackXParams &p, cudaStream_t st) {
    return launch_pdl(pack_x_kernel, dim3(p.rows), dim3(256), 0, st, true, p);
}

cudaError_t bp_router(const RouterArgs &args, cudaStream_t st) {
    const RouterParams &p = args.p;
    return launch_pdl(router_gemm_kernel, dim3(p.experts / 128, (p.tokens + kRouterTileTokens - 1) / kRouterTileTokens, p.splits),
                      dim3(128), kRouterSmem, st, true, args);
}

uint32_t bp_route_blocks(uint32_t tokens) {
    const uint32_t tpb = bp_tokens_per_block(tokens);
    return (tokens + tpb - 1) / tpb;
}

cudaError_t bp_route(const RouteParams &p, cudaStream_t st) {
    if (p.tokens <= kSmallRoute) return launch_pdl(route_small_kernel, dim3(1), dim3(1024), 0, st, true, p);
    const dim3 grid(bp_route_blocks(p.tokens));
    const bool eight = bp_tokens_per_block(p.tokens) == 8, one_segment = p.tokens <= kRouteShort;
    cudaError_t e = one_segment ? launch_pdl(route_kernel<8, false>, grid, dim3(256), 0, st, true, p)
                    : eight     ? launch_pdl(route_kernel<8, true>, grid, dim3(256), 0, st, true, p)
                                : launch_pdl(route_kernel<32, true>, grid, dim3(1024), 0, st, true, p);
    if (e != cudaSuccess) return e;
    return one_segment ? launch_pdl(route_scatter_kernel<false>, grid, dim3(256), 0, st, true, p)
                       : launch_pdl(route_scatter_kernel<true>, grid, dim3(256), 0, st, true, p);
}

cudaError_t bp_pack_acts(const PackActsParams &p, cudaStream_t st) {
    return launch_pdl(pack_acts_kernel, dim3((p.rows + p.rows2 + 7) / 8), dim3(256), 0, st, true, p);
}

cudaError_t bp_combine(const CombineRowsParams &in, uint32_t out_dtype, cudaStream_t st) {
    CombineRowsParams p = in;
    p.aligned = ((reinterpret_cast<uintptr_t>(p.y) | reinterpret_cast<uintptr_t>(p.hidden) | reinterpret_cast<uintptr_t>(p.hidden_delta) |
                  reinterpret_cast<uintptr_t>(p.partial_y)) & 15u) == 0 ? 1u : 0u;
    const bool half_rows = p.x_next == nullptr && out_dtype == OUT_F16 && p.partial_half;
    const dim3 grid(std::min(p.tokens, p.sms * kCombineBlocks[half_rows ? 0 : 1])), block(256);
    if (p.x_next != nullptr)
        return out_dtype == OUT_F16 ? launch_pdl(combine_rows_kernel<OUT_F16, OUT_F32, true>, grid, block, 0, st, true, p)
                                    : launch_pdl(combine_rows_kernel<OUT_F32, OUT_F32, true>, grid, block, 0, st, true, p);
    if (out_dtype == OUT_F16) {
        if (p.partial_half) return launch_pdl(combine_rows_kernel<OUT_F16, OUT_F16, false>, grid, block, 0, st, true, p);
        return launch_pdl(combine_rows_kernel<OUT_F16, OUT_F32, false>, grid, block, 0, st, true, p);
    }
    return launch_pdl(combine_rows_kernel<OUT_F32, OUT_F32, false>, grid, block, 0, st, true, p);
}

cudaError_t bp_set_wait_limit(unsigned long long ns) { return cudaMemcpyToSymbol(g_wait_limit_ns, &ns, sizeof(ns)); }

}  // namespace nvmai
