// Launchers of the batched path: see batch_path.h.
#include "batch_path.h"

#include <algorithm>
#include <type_traits>

#include "batch_rows.cuh"
#include "expert_gemm.cuh"
#include "launch.h"

namespace nvmai {

namespace {
constexpr size_t kMaxBlockSmem = 227 * 1024;
}

EgPlan eg_plan(EgParams &p, int phase, uint32_t want_cap) {
    const uint32_t n_main = p.kdim / 64, n_kb = n_main + bp_extra_cols(p.kdim, phase == 0 ? 1 : 2) / 64;
    const size_t fixed = 2048 + (size_t)kEgChunks * kEgChunkBytes;           // alignment slack, barriers, code ring
    p.meta_slot_bytes = 128 * n_main * 4;
    p.meta_slots = (size_t)4 * p.meta_slot_bytes <= 64 * 1024 ? 4 : 2;
    const size_t meta = ((size_t)p.meta_slots * p.meta_slot_bytes + 1023) & ~(size_t)1023;
    if (fixed + meta + 2 * 2048 > kMaxBlockSmem) return EgPlan{0, 0};
    const size_t avail = kMaxBlockSmem - fixed - meta;
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
    p.row_slot_bytes = cap * 128;
    p.row_slots = (uint32_t)std::min<size_t>(kEgMaxRowSlots, avail / p.row_slot_bytes);
    p.row_ring_off = (uint32_t)(1024 + (size_t)kEgChunks * kEgChunkBytes + meta);
    if (phase == 0) {
        p.acc_slots = std::min(kEgMaxAcc, kEgAccCols / (2 * cap));
        p.acc_stride = kEgAccCols / p.acc_slots / 32 * 32;
        p.acc_tile_off = p.acc_stride / 2;
    } else {
        p.acc_slots = std::min(kEgMaxAcc, kEgAccCols / cap);
        p.acc_stride = kEgAccCols / p.acc_slots / 16 * 16;
        p.acc_tile_off = 0;
    }
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
    const dim3 grid(bp_route_blocks(p.tokens));
    cudaError_t e = launch_pdl(route_kernel, grid, dim3(256), 0, st, true, p);
    if (e != cudaSuccess) return e;
    return launch_pdl(route_scatter_kernel, grid, dim3(256), 0, st, true, p);
}

cudaError_t bp_pack_acts(const PackActsParams &p, cudaStream_t st) {
    return launch_pdl(pack_acts_kernel, dim3((p.rows + p.rows2 + 7) / 8), dim3(256), 0, st, true, p);
}

cudaError_t bp_combine(const CombineRowsParams &in, uint32_t out_dtype, cudaStream_t st) {
    CombineRowsParams p = in;
    p.aligned = ((reinterpret_cast<uintptr_t>(p.y) | reinterpret_cast<uintptr_t>(p.hidden) | reinterpret_cast<uintptr_t>(p.hidden_delta) |
                  reinterpret_cast<uintptr_t>(p.partial_y)) & 15u) == 0 ? 1u : 0u;
    const dim3 grid(p.tokens), block(256);
    if (out_dtype == OUT_F16) {
        if (p.partial_half) return launch_pdl(combine_rows_kernel<OUT_F16, OUT_F16>, grid, block, 0, st, true, p);
        return launch_pdl(combine_rows_kernel<OUT_F16, OUT_F32>, grid, block, 0, st, true, p);
    }
    return launch_pdl(combine_rows_kernel<OUT_F32, OUT_F32>, grid, block, 0, st, true, p);
}

cudaError_t bp_set_wait_limit(unsigned long long ns) { return cudaMemcpyToSymbol(g_wait_limit_ns, &ns, sizeof(ns)); }

}  // namespace nvmai
