// The kernels around the grouped expert GEMMs: x rows packed for the tensor cores, the dense router, top-k with the
// grouping of the (token, expert) pairs, activation rows of the wide-range mode, and the per-token reduction.
#pragma once

#include "batch_path.h"
#include "decode_kernels.cuh"
#include "tcgen05.cuh"

namespace nvmai {

constexpr uint32_t kBpNotLocal = 0xFFFFFFFFu;

// ---- x rows ---------------------------------------------------------------------------------
// One block per row, 8 values per thread: the row in the weights' K order, the sums of its 64-value groups as fp16
// hi + lo behind it ([hi | lo | hi | 0], see expert_gemm.cuh), and the scalar gate of the row (the row is in registers
// anyway; as a launch of its own the gate took 17-31 us).
__global__ void __launch_bounds__(256) pack_x_kernel(PackXParams p) {
    __shared__ float wsum[8];
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const size_t row = blockIdx.x;
    const uint32_t extra = bp_extra_cols(p.n, 1), G = p.n / 64u;
    const size_t stride = (size_t)p.n + extra;
    __half *dst = p.dst + row * stride, *dst2 = p.dst2 != nullptr ? p.dst2 + row * stride : nullptr;
    float gate = 0.0f;
    for (uint32_t base = 0; base < p.n; base += 2048u) {
        const uint32_t i8 = base + tid * 8u;
        float part = 0.0f;
        if (i8 < p.n) {
            const uint4 q = *reinterpret_cast<const uint4 *>(p.x + row * p.n + i8);
            // natural (0,1)(2,3)(4,5)(6,7) -> (0,4)(1,5)(2,6)(3,7), the order of bp_k_order
            const uint4 perm = make_uint4(__byte_perm(q.x, q.z, 0x5410), __byte_perm(q.x, q.z, 0x7632),
                                          __byte_perm(q.y, q.w, 0x5410), __byte_perm(q.y, q.w, 0x7632));
            if (p.dst != nullptr) *reinterpret_cast<uint4 *>(dst + i8) = p.permute ? perm : q;
            if (dst2 != nullptr) *reinterpret_cast<uint4 *>(dst2 + i8) = p.permute ? q : perm;
            const __half2 *h = reinterpret_cast<const __half2 *>(&q);
            float f[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 t = __half22float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
#pragma unroll
            for (int i = 0; i < 8; ++i) part += f[i];
            if (p.gate_row != nullptr) {
                const uint4 w = __ldg(reinterpret_cast<const uint4 *>(p.gate_row + i8));
                const __half2 *wh = reinterpret_cast<const __half2 *>(&w);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 t = __half22float2(wh[i]);
                    gate = fmaf(t.x, f[2 * i], gate);
                    gate = fmaf(t.y, f[2 * i + 1], gate);
                }
            }
        }
        part += __shfl_xor_sync(0xffffffffu, part, 1);       // a group = 8 neighbouring lanes
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        part += __shfl_xor_sync(0xffffffffu, part, 4);
        if (p.dst != nullptr && i8 < p.n && (lane & 7u) == 0u) {
            const float sum = part * kBpSumScale;
            const __half hi = __float2half_rn(sum), lo = __float2half_rn(sum - __half2float(hi));
            const uint32_t g = i8 / 64u;
            dst[p.n + g] = hi; dst[p.n + G + g] = lo; dst[p.n + 2u * G + g] = hi;
            if (dst2 != nullptr) { dst2[p.n + g] = hi; dst2[p.n + G + g] = lo; dst2[p.n + 2u * G + g] = hi; }
        }
    }
    for (uint32_t i = 3u * G + tid; p.dst != nullptr && i < extra; i += 256u) {
        dst[p.n + i] = __float2half_rn(0.0f);
        if (dst2 != nullptr) dst2[p.n + i] = __float2half_rn(0.0f);
    }
    if (p.gate_row != nullptr) {
        gate = warp_sum(gate);
        if (lane == 0) wsum[tid >> 5] = gate;
        __syncthreads();
        if (tid == 0) {
            float tot = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) tot += wsum[i];
            p.gate_val[row] = p.out_half ? round_f16(tot) : round11(tot);
        }
    }
}

// ---- dense router ---------------------------------------------------------------------------
// logits[split][token][expert]: 128 router rows x 64 token rows per block, K split over blockIdx.z so that a small
// batch still spreads over the chip (one block per 256 tokens took 20-29 us at any batch size).  Products of two fp16
// values are exact in fp32: only the order of the additions differs from the decode router's.  That order is the same
// for any number of splits, so a row's logits do not depend on the rows beside it: K always adds up in four quarters,
// ((q0 + q1) + q2) + q3, a block keeping each of its quarters in an accumulator of its own.  The first block hands over the
// sum of its quarters, the others each quarter: 1, 3 or 4 terms for 1, 2 or 4 splits (bp_router_terms).
constexpr uint32_t kRouterStages = 4;
constexpr uint32_t kRouterStageBytes = 128 * 128 + kRouterTileTokens * 128;
constexpr size_t kRouterSmem = 2048 + kRouterStages * kRouterStageBytes;
struct RouterBarriers { uint64_t full[kRouterStages], empty[kRouterStages], done; uint32_t tmem_slot; };

__global__ void __launch_bounds__(128) router_gemm_kernel(const __grid_constant__ RouterArgs args) {
    extern __shared__ unsigned char rt_smem_raw[];
    const RouterParams &p = args.p;
    const uint32_t raw = smem_addr(rt_smem_raw), base = (raw + 1023u) & ~1023u;
    RouterBarriers *bars = reinterpret_cast<RouterBarriers *>(rt_smem_raw + (base - raw));
    const uint32_t ring = base + 1024u;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < kRouterStages; ++i) { mbar_init(&bars->full[i], 1); mbar_init(&bars->empty[i], 1); }
        mbar_init(&bars->done, 1);
        mbar_fence_init();
    }
    if (warp == 1) { tmem_alloc(&bars->tmem_slot, kRouterParts * kRouterTileTokens); tmem_relinquish(); }      // (two blocks per SM)
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&bars->tmem_slot);
    // x was complete before the kernel in front of this one (which packs it) could pass its own wait
    const uint32_t n_kb = p.kdim / 64u / p.splits, kb0 = blockIdx.z * n_kb;
    const uint32_t quarters = kRouterParts / p.splits, quarter_kb = p.kdim / 64u / kRouterParts;      // this block's
    const uint32_t e0 = blockIdx.x * 128u, t0 = blockIdx.y * kRouterTileTokens;
    bool ok = *reinterpret_cast<volatile unsigned int *>(p.status) == 0u;
    ok = __syncthreads_and(ok);
    if (warp == 0) {
        if (elect_one()) {
            for (uint32_t k = 0; k < n_kb && ok; ++k) {
                const uint32_t s = k % kRouterStages, st = ring + s * kRouterStageBytes;
                ok = mbar_wait(&bars->empty[s], ((k / kRouterStages) & 1u) ^ 1u, p.status);
                if (!ok) break;
                mbar_expect_tx(&bars->full[s], kRouterStageBytes);
                tma_load_2d(st, &args.w, (kb0 + k) * 64u, e0, &bars->full[s]);
                tma_load_2d(st + 128u * 128u, &args.x, (kb0 + k) * 64u, t0, &bars->full[s]);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_f16(128u, kRouterTileTokens);
            uint32_t acc = tmem, in_quarter = 0;
            for (uint32_t k = 0; k < n_kb && ok; ++k) {
                const uint32_t s = k % kRouterStages, st = ring + s * kRouterStageBytes;
                ok = mbar_wait(&bars->full[s], (k / kRouterStages) & 1u, p.status);
                if (!ok) break;
                tc_fence_after_sync();
                const uint64_t da = umma_desc_sw128(st), db = umma_desc_sw128(st + 128u * 128u);
#pragma unroll
                for (uint32_t j = 0; j < 4u; ++j) umma_f16_ss(acc, da + 2u * j, db + 2u * j, idesc, (in_quarter | j) != 0u);
                umma_commit(&bars->empty[s]);
                if (++in_quarter == quarter_kb) { in_quarter = 0; acc += kRouterTileTokens; }
            }
            if (ok) umma_commit(&bars->done);
        }
        __syncwarp();
    }
    if (ok) ok = mbar_wait(&bars->done, 0, p.status);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
        tc_fence_after_sync();
        const uint32_t term = blockIdx.z == 0u ? 0u : p.splits == 2u ? 1u : blockIdx.z;
        const size_t term_step = (size_t)p.tokens * p.experts;
        float *out = p.logits + term * term_step + (size_t)t0 * p.experts + e0 + warp * 32u + lane;
        for (uint32_t cb = 0; cb < kRouterTileTokens && t0 + cb < p.tokens; cb += 8u) {
            uint32_t r[kRouterParts][8];
#pragma unroll
            for (uint32_t q = 0; q < kRouterParts; ++q)
                if (q < quarters) tmem_ld8(tmem + ((warp * 32u) << 16) + q * kRouterTileTokens + cb, r[q]);
            tmem_ld_wait();
            float *at = out + (size_t)cb * p.experts;
#pragma unroll
            for (uint32_t q = 0; q < kRouterParts; ++q) {
                if (q >= quarters) break;
                if (q != 0u) {
                    if (blockIdx.z != 0u) at += term_step;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (blockIdx.z == 0u) r[q][i] = __float_as_uint(__uint_as_float(r[q - 1u][i]) + __uint_as_float(r[q][i]));
                }
                if (blockIdx.z == 0u && q + 1u < quarters) continue;
#pragma unroll
                for (uint32_t i = 0; i < 8u; ++i)
                    if (t0 + cb + i < p.tokens) at[(size_t)i * p.experts] = __uint_as_float(r[q][i]);
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kRouterParts * kRouterTileTokens);
    pdl_wait();                     // the kernel after this one relies on the one before it being complete
    pdl_launch_dependents();
}

// ---- top-k and grouping -----------------------------------------------------------------------
// Tokens (and warps) per block: 8 up to 1024 tokens, 32 above, so that a chunk of 4096 is one wave of 128 blocks.
__host__ __device__ constexpr uint32_t bp_tokens_per_block(uint32_t tokens) { return tokens <= 1024u ? 8u : 32u; }
constexpr uint32_t kRouteShort = 768;      // rows of calls that have one segment by their size (see route_kernel)
static_assert(bp_tokens_per_block(kRouteShort) == 8u && kRouteShort <= 8u * kRouteSegment, "blocks of eight tokens, one segment");

// Expert e's work items in list j: its rows split evenly over them (two items of 70 instead of 128 + 12).
__device__ __forceinline__ void write_items(const RouteParams &p, int j, uint32_t e, uint32_t rows, uint32_t items, uint32_t first_row,
                                            uint32_t first_item) {
    const uint32_t even = items ? rows / items : 0u, extra = items ? rows % items : 0u;
    for (uint32_t i = 0; i < items; ++i)
        p.work[j][first_item + i] = WorkItem{e, first_row + i * even + min(i, extra), even + (i < extra ? 1u : 0u), 0u};
}

__device__ __forceinline__ uint32_t item_count(const RouteParams &p, int j, uint32_t rows, uint32_t heavy) {
    return (rows > heavy) == (j < 2) ? (rows + p.cap[j] - 1u) / p.cap[j] : 0u;
}
// whole block, `rows` = the rows of expert threadIdx.x: the limit that applies (see RouteParams); ends in sync
__device__ __forceinline__ uint32_t heavy_limit(const RouteParams &p, uint32_t rows) {
    __shared__ uint32_t heavy_pairs;
    if (p.heavy == 0u || p.heavy == ~0u) {
        if (threadIdx.x == 0) { p.shared_on[0] = p.heavy == 0u; p.shared_on[1] = p.heavy != 0u; }
        return p.heavy;
    }
    if (threadIdx.x == 0) heavy_pairs = 0u;
    __syncthreads();
    if (rows > p.heavy) atomicAdd(&heavy_pairs, rows);
    __syncthreads();
    const bool many = heavy_pairs >= p.heavy_min;
    if (threadIdx.x == 0) { p.shared_on[0] = many; p.shared_on[1] = !many; }
    return many ? p.heavy : ~0u;
}

// v[i] = logit of expert lane + 32 i: its terms added in order, all 32 loads in flight
__device__ __forceinline__ void add_terms(float (&v)[kMaxExperts / 32], const RouteParams &p, uint32_t tok, uint32_t lane) {
    static_assert(kRouterParts == 4, "the sum has four terms");
    float a[4][kMaxExperts / 32];
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k)
#pragma unroll
        for (int i = 0; i < kMaxExperts / 32; ++i) {
            const uint32_t e = lane + 32u * i;
            a[k][i] = e < p.E && k < p.terms ? __ldcg(p.logits + ((size_t)k * p.tokens + tok) * p.E + e) : 0.0f;
        }
#pragma unroll
    for (int i = 0; i < kMaxExperts / 32; ++i)
        if (lane + 32u * i < p.E) v[i] = ((a[0][i] + a[1][i]) + a[2][i]) + a[3][i];
}

// Router semantics of router_topk_select_k8 (moe.metal:233-285); the pairs end up in (expert, token, rank) order, as
// PrefillMoEGrouping.groupTokenExpertPairs has them (PrefillMoEGrouping.swift:90-192).  A warp per token.  The whole chip
// waits while the last block makes the work lists, so that block gets by with 256 totals a segment of 128 blocks, which the
// blocks have added up with atomics; where a block's own pairs begin, the scatter works out from the counts of the blocks before
// it in its segment: one segment up to 4096 rows; counts of all blocks in front would grow with the square of the rows (256 /
// 128 wide, 262,144 rows: 5519 us, 4940 with segments; 4096 rows 112 either way).  (With four tokens per warp and a last block that
// scanned every block's counts, 4096 rows took 33 us from the router's end to this kernel's, 1531 rows 29, 256 rows 14.)
// LONG: with segments; up to kRouteShort rows without, which their loop over the counts leaves at 32 registers instead of 80 (whole
// call, 256 skewed rows 99.2 / 100.2 us without / with, 600 143.1 / 143.5; 1000 rows of 256 / 128 68.0 / 66.6, 1500 76.7 / 75.4).
template <int WARPS, bool LONG>
__global__ void __launch_bounds__(WARPS * 32) route_kernel(RouteParams p) {
    static_assert(WARPS * 32 >= kMaxExperts, "a thread per expert");
    __shared__ uint32_t hist[kMaxExperts];
    __shared__ uint32_t warp_tot[4][kMaxExperts / 32];
    __shared__ bool last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < kMaxExperts) hist[tid] = 0;
    pdl_wait();
    pdl_launch_dependents();
    __syncthreads();
    const uint32_t tok = blockIdx.x * WARPS + warp;
    if (tok < p.tokens) {
        if (p.logits != nullptr) {
            float v[kMaxExperts / 32];
#pragma unroll
            for (int i = 0; i < kMaxExperts / 32; ++i) v[i] = lane + 32u * i < p.E ? 0.0f : -INFINITY;
            add_terms(v, p, tok, lane);
            topk_softmax_warp_vals(v, (int)p.E, (int)p.K, p.pes, p.idx + (size_t)tok * p.K, p.w + (size_t)tok * p.K);
        }
        if ((uint32_t)lane < p.K) {
            const uint32_t g = min(p.idx[(size_t)tok * p.K + lane], p.E - 1u);
            const uint32_t e = p.expert_map != nullptr ? p.expert_map[g] : g;
            if (e != kBpNotLocal) atomicAdd(&hist[e], 1u);
        }
    }
    __syncthreads();
    if (tid < kMaxExperts && hist[tid] != 0u) atomicAdd(p.totals + (LONG ? blockIdx.x / kRouteSegment * kMaxExperts : 0u) + tid, hist[tid]);
    if (tid < kMaxExperts / 4)      // at most 32 * kMaxTopK pairs of an expert (a caller's list may repeat one)
        reinterpret_cast<uint2 *>(p.block_hist)[(size_t)blockIdx.x * (kMaxExperts / 4) + tid] =
            make_uint2(hist[4 * tid] | hist[4 * tid + 1] << 16, hist[4 * tid + 2] | hist[4 * tid + 3] << 16);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(p.counter, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!last) return;
    // thread e owns expert e: exclusive scans of the pairs and of the launches' work items
    __threadfence();
    if (tid == 0) *p.counter = 0u;
    uint32_t total = 0;
    if (tid < kMaxExperts) {
        total = __ldcg(p.totals + tid);
        p.totals[tid] = 0u;
        if constexpr (LONG)
            for (uint32_t i = kMaxExperts + tid; i < bp_route_segments(gridDim.x) * kMaxExperts; i += kMaxExperts) {
                const uint32_t n = __ldcg(p.totals + i);
                p.totals[i] = 0u;
                p.first[i] = total;
                total += n;
            }
    }
    const uint32_t heavy = heavy_limit(p, total);
    uint32_t mine[4] = {}, pre[4];
    if (tid < kMaxExperts) {
        mine[0] = total;
#pragma unroll
        for (int j = 0; j < 3; ++j) mine[1 + j] = item_count(p, j, total, heavy);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            pre[j] = mine[j];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, pre[j], o);
                if (lane >= o) pre[j] += v;
            }
            if (lane == 31) warp_tot[j][warp] = pre[j];
        }
    }
    __syncthreads();
    if (tid >= kMaxExperts) return;
    uint32_t all[4] = {};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        pre[j] -= mine[j];
        for (int w = 0; w < kMaxExperts / 32; ++w) {
            if (w < warp) pre[j] += warp_tot[j][w];
            all[j] += warp_tot[j][w];
        }
    }
    p.first[tid] = pre[0];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        write_items(p, j, tid, total, mine[1 + j], pre[0], pre[1 + j]);
        if (tid == 0) p.n_work[j][0] = all[1 + j];
    }
}

// stable scatter of a block's pairs
template <bool LONG>
__global__ void __launch_bounds__(256) route_scatter_kernel(RouteParams p) {
    __shared__ uint16_t cnt[8][kMaxExperts];
    __shared__ uint32_t before[4][kMaxExperts];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int w = 0; w < 8; ++w) cnt[w][tid] = 0;
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t tpb = bp_tokens_per_block(p.tokens), pairs = tpb * p.K, first = blockIdx.x * pairs;     // <= 256 pairs
    const uint32_t i = first + tid, P = p.tokens * p.K;
    uint32_t e = kBpNotLocal;
    const bool mine = (uint32_t)tid < pairs && i < P;
    if (mine) {
        const uint32_t g = min(p.idx[i], p.E - 1u);
        e = p.expert_map != nullptr ? p.expert_map[g] : g;
    }
    // the pairs of the segment's blocks in front: a quarter of the blocks a thread, four experts each, 32 blocks' counts in flight
    const uint32_t segment = LONG ? blockIdx.x / kRouteSegment : 0u;
    {
        constexpr uint32_t kBatch = kRouteSegment / 4u;
        const uint32_t part = tid >> 6, quad = tid & 63;
        uint32_t n[4] = {};
        auto add = [&](uint32_t b0) {
            uint2 c[kBatch], sum = make_uint2(0u, 0u);
#pragma unroll
            for (uint32_t k = 0; k < kBatch; ++k)
                c[k] = b0 + 4u * k < blockIdx.x
                           ? __ldcg(reinterpret_cast<const uint2 *>(p.block_hist) + (size_t)(b0 + 4u * k) * (kMaxExperts / 4) + quad) : make_uint2(0u, 0u);
#pragma unroll
            for (uint32_t k = 0; k < kBatch; ++k) { sum.x += c[k].x; sum.y += c[k].y; }      // (32 x 256 fits 16 bits)
            n[0] += sum.x & 0xFFFFu; n[1] += sum.x >> 16; n[2] += sum.y & 0xFFFFu; n[3] += sum.y >> 16;
        };
        if constexpr (LONG) {
            const uint32_t b0 = segment * kRouteSegment + part;
            if (b0 < blockIdx.x) add(b0);
        } else {
            for (uint32_t b0 = part; b0 < blockIdx.x; b0 += 4u * kBatch) add(b0);
        }
        *reinterpret_cast<uint4 *>(&before[part][4 * quad]) = make_uint4(n[0], n[1], n[2], n[3]);
    }
    const bool live = e != kBpNotLocal;
    if (mine && !live) p.inv[i] = kBpNotLocal;
    const uint32_t peers = __match_any_sync(0xffffffffu, e);
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    __syncthreads();
    if (live && rank == 0u) cnt[warp][e] = (uint16_t)__popc(peers);
    __syncthreads();
    if (live) {
        uint32_t pos = __ldcg(p.first + e) + rank;
        if (LONG && segment != 0u) pos += __ldcg(p.first + segment * kMaxExperts + e);
#pragma unroll
        for (int q = 0; q < 4; ++q) pos += before[q][e];
        for (int w = 0; w < warp; ++w) pos += cnt[w][e];
        p.sorted_pair[pos] = i;
        p.inv[i] = pos;
    }
}

// The same in one block for up to kSmallRoute tokens: histogram, scan and scatter stay in shared memory (two launches
// and two trips through global memory less: 13 rows 12.4 + 3.2 us as two launches).
__global__ void __launch_bounds__(1024) route_small_kernel(RouteParams p) {
    __shared__ uint32_t hist[kMaxExperts], first[kMaxExperts];
    __shared__ uint16_t cnt[8][kMaxExperts];                  // per warp of pairs, at most 256 pairs
    __shared__ uint16_t pair_expert[kSmallRoute * kMaxTopK];
    __shared__ uint32_t warp_tot[4][kMaxExperts / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < kMaxExperts) {
        hist[tid] = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) cnt[w][tid] = 0;
    }
    pdl_wait();
    pdl_launch_dependents();
    __syncthreads();
    for (uint32_t tok = warp; tok < p.tokens; tok += 32u) {
        if (p.logits != nullptr) {
            float v[kMaxExperts / 32];
#pragma unroll
            for (int i = 0; i < kMaxExperts / 32; ++i) v[i] = lane + 32u * i < p.E ? 0.0f : -INFINITY;
            add_terms(v, p, tok, lane);
            topk_softmax_warp_vals(v, (int)p.E, (int)p.K, p.pes, p.idx + (size_t)tok * p.K, p.w + (size_t)tok * p.K);
        }
        if ((uint32_t)lane < p.K) {
            const uint32_t g = min(p.idx[(size_t)tok * p.K + lane], p.E - 1u);
            const uint32_t e = p.expert_map != nullptr ? p.expert_map[g] : g;
            pair_expert[tok * p.K + lane] = (uint16_t)(e == kBpNotLocal ? 0xFFFFu : e);
            if (e != kBpNotLocal) atomicAdd(&hist[e], 1u);
        }
    }
    __syncthreads();
    const uint32_t P = p.tokens * p.K;
    const uint32_t e = (uint32_t)tid < P ? pair_expert[tid] : 0xFFFFu;
    const bool live = e != 0xFFFFu;
    const uint32_t peers = __match_any_sync(0xffffffffu, e);
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    if (live && rank == 0u) cnt[warp][e] = (uint16_t)__popc(peers);
    const uint32_t heavy = heavy_limit(p, tid < kMaxExperts ? hist[tid] : 0u);
    uint32_t total = 0, mine[4] = {}, pre[4] = {};
    if (tid < kMaxExperts) {
        total = hist[tid];
        mine[0] = total;
#pragma unroll
        for (int j = 0; j < 3; ++j) mine[1 + j] = item_count(p, j, total, heavy);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            pre[j] = mine[j];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, pre[j], o);
                if (lane >= o) pre[j] += v;
            }
            if (lane == 31) warp_tot[j][warp] = pre[j];
        }
    }
    __syncthreads();
    if (tid < kMaxExperts) {
        uint32_t all[4] = {};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            pre[j] -= mine[j];
            for (int w = 0; w < kMaxExperts / 32; ++w) {
                if (w < warp) pre[j] += warp_tot[j][w];
                all[j] += warp_tot[j][w];
            }
        }
        first[tid] = pre[0];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            write_items(p, j, tid, total, mine[1 + j], pre[0], pre[1 + j]);
            if (tid == 0) p.n_work[j][0] = all[1 + j];
        }
    }
    __syncthreads();
    if (live) {
        uint32_t pos = first[e] + rank;
        for (int w = 0; w < warp; ++w) pos += cnt[w][e];
        p.sorted_pair[pos] = tid;
        p.inv[tid] = pos;
    } else if ((uint32_t)tid < P) {
        p.inv[tid] = kBpNotLocal;
    }
}

// ---- wide-range activation rows ------------------------------------------------------------------
// One warp per row: fp32 rows scaled by a power of two that brings the row's largest magnitude to [2^14, 2^15), so
// that the fp16 copy neither overflows nor loses its small entries to subnormals (the down GEMM's epilogue multiplies
// the factor back), in the down weights' K order, with half-group sums.
__global__ void __launch_bounds__(256) pack_acts_kernel(PackActsParams p) {
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t row = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    const bool second = row >= p.rows;
    const uint32_t r = second ? row - p.rows : row;
    if (second && r >= p.rows2) return;
    const uint32_t n = second ? p.n2 : p.n, permute = second ? p.permute2 : p.permute;
    const float *src = (second ? p.src2 : p.src) + (size_t)r * n;
    const uint32_t extra = bp_extra_cols(n, 2), slots = n / 32u;
    __half *dst = (second ? p.dst2 : p.dst) + (size_t)r * (n + extra);
    constexpr int kKeep = 4;                 // 256 values per pass; up to 1024 stay in registers between the two passes
    float4 keep[kKeep][2];
    float m = 0.0f;
    auto load = [&](uint32_t i8, float4 (&v)[2]) {
        const float4 *s4 = reinterpret_cast<const float4 *>(src + i8);
        v[0] = s4[0]; v[1] = s4[1];
    };
    auto peak = [&](const float4 (&v)[2]) {
        const float *f = reinterpret_cast<const float *>(v);
#pragma unroll
        for (int i = 0; i < 8; ++i) { const float a = fabsf(f[i]); m = (a <= 3.0e38f && a > m) ? a : m; }   // not inf, not NaN
    };
#pragma unroll
    for (int k = 0; k < kKeep; ++k) {
        const uint32_t i8 = k * 256u + lane * 8u;
        if (i8 < n) { load(i8, keep[k]); peak(keep[k]); }
    }
    for (uint32_t i8 = kKeep * 256u + lane * 8u; i8 < n; i8 += 256u) { float4 v[2]; load(i8, v); peak(v); }
#pragma unroll
    for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    int e = 0;
    if (m > 0.0f) frexpf(m, &e);                          // m = f * 2^e, f in [0.5, 1)
    const int shift = m > 0.0f ? 15 - e : 0;
    const float mul = ldexpf(1.0f, shift);
    if (lane == 0) (second ? p.row_scale2 : p.row_scale)[r] = ldexpf(1.0f, -shift);
    auto put = [&](uint32_t base, const float4 (&v)[2]) {
        const uint32_t i8 = base + lane * 8u;
        float part = 0.0f;
        if (i8 < n) {
            const float *f = reinterpret_cast<const float *>(v);
            __half h[8], o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) { h[i] = __float2half_rn(f[i] * mul); part += __half2float(h[i]); }
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = permute ? h[bp_k_order(i)] : h[i];
            *reinterpret_cast<uint4 *>(dst + i8) = *reinterpret_cast<const uint4 *>(o);
        }
        part += __shfl_xor_sync(0xffffffffu, part, 1);     // half a group = 4 neighbouring lanes
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        if (i8 < n && (lane & 3u) == 0u) {
            const float sum = part * kBpSumScale;
            const __half hi = __float2half_rn(sum), lo = __float2half_rn(sum - __half2float(hi));
            const uint32_t s = i8 / 32u;
            dst[n + s] = hi; dst[n + slots + s] = lo; dst[n + 2u * slots + s] = hi;
        }
    };
#pragma unroll
    for (int k = 0; k < kKeep; ++k)
        if (k * 256u < n) put(k * 256u, keep[k]);
    for (uint32_t base = kKeep * 256u; base < n; base += 256u) {
        float4 v[2] = {};
        if (base + lane * 8u < n) load(base + lane * 8u, v);
        put(base, v);
    }
}

// ---- per-token reduction ----------------------------------------------------------------------
// aligned: the caller's pointer is 16-byte aligned (i always is a multiple of 8)
template <int OUT> __device__ __forceinline__ void load_out8(const void *p, size_t i, float (&v)[8], bool aligned = true) {
    if (!aligned) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = load_out<OUT>(p, i + k);
    } else if (OUT == OUT_F16) {
        const uint4 q = *reinterpret_cast<const uint4 *>(static_cast<const __half *>(p) + i);
        const __half2 *h = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
        for (int k = 0; k < 4; ++k) { const float2 t = __half22float2(h[k]); v[2 * k] = t.x; v[2 * k + 1] = t.y; }
    } else {
        const float4 *f = reinterpret_cast<const float4 *>(static_cast<const float *>(p) + i);
        const float4 a = f[0], b = f[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}
template <int OUT> __device__ __forceinline__ void store_out8(void *p, size_t i, const float (&v)[8], bool aligned = true) {
    if (!aligned) {
#pragma unroll
        for (int k = 0; k < 8; ++k) store_out<OUT>(p, i + k, v[k]);
    } else if (OUT == OUT_F16) {
        uint4 q;
        uint32_t *w = reinterpret_cast<uint32_t *>(&q);
#pragma unroll
        for (int k = 0; k < 4; ++k) { const __half2 h = __floats2half2_rn(v[2 * k], v[2 * k + 1]); w[k] = *reinterpret_cast<const uint32_t *>(&h); }
        *reinterpret_cast<uint4 *>(static_cast<__half *>(p) + i) = q;
    } else {
        float4 *f = reinterpret_cast<float4 *>(static_cast<float *>(p) + i);
        f[0] = make_float4(v[0], v[1], v[2], v[3]);
        f[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// 8 values of a partial row as they were loaded
template <int PART> struct Part8 {
    uint4 q[PART == OUT_F16 ? 1 : 2];
    __device__ __forceinline__ void load(const void *p, size_t i) {
        const uint4 *s = PART == OUT_F16 ? reinterpret_cast<const uint4 *>(static_cast<const __half *>(p) + i)
                                         : reinterpret_cast<const uint4 *>(static_cast<const float *>(p) + i);
#pragma unroll
        for (int k = 0; k < (PART == OUT_F16 ? 1 : 2); ++k) q[k] = s[k];
    }
    __device__ __forceinline__ float at(int k) const {      // k: a constant
        const uint32_t *w = reinterpret_cast<const uint32_t *>(q);
        if (PART == OUT_F32) return __uint_as_float(w[k]);
        const __half2 h = *reinterpret_cast<const __half2 *>(&w[k >> 1]);
        return (k & 1) ? __high2float(h) : __low2float(h);
    }
};

// A block walks every gridDim-th token, 8 values per thread; every slot's partial row is requested before any is used (the version that
// walked the slots value by value took 19-23 us for any batch).  Slot order, so the result does not depend on the
// grouping.  PART: type of the partial rows.  Prefill rounding (prefill.metal:437-458, RealForwardRunner.swift:3560-3569):
// every partial is rounded to the output type, h2 = out(sum_r fma(w, partial)) on its own, and the residual takes two
// steps: hidden = out(out(hidden + h1) + h2).  Decode order: one rounding of h1 + sum, one residual add.
// NORM: the row's RMS-normalised form is stored as the next block's input.  Its own variant: with the norm's code in it the
// plain reduction of 1531 rows took 47 us instead of 26; with the partial rows kept as loaded (80 registers, three blocks
// per SM, for half rows) it takes 20, 46 at 4096 rows.
// The grid is what is resident at once; a row's positions and weights are requested while the row before it is added up, the
// first one's before the wait: with a block per token and all of it behind the wait, a stack of 5 rows took 163.7 us instead of
// 159.3, 13 rows 60.0 instead of 58.2, the reduction of 4096 rows 57 instead of 54.
constexpr int kCombineBlocks[2] = {3, 2};      // resident per SM: half, fp32 partial rows
template <int OUT, int PART, bool NORM>
__global__ void __launch_bounds__(256, kCombineBlocks[PART == OUT_F16 ? 0 : 1]) combine_rows_kernel(CombineRowsParams p) {
    __shared__ uint32_t pos_of[2][kMaxTopK];
    __shared__ float weight_of[2][kMaxTopK];
    __shared__ float row[NORM ? kBpNormRow : 1];
    __shared__ float wsum[8];
    uint32_t next_pos = 0;
    float next_weight = 0.0f;
    auto request = [&](uint32_t t) {
        if (threadIdx.x >= p.K) return;
        next_pos = p.inv[(size_t)t * p.K + threadIdx.x];
        next_weight = __half2float(p.routing_w[(size_t)t * p.K + threadIdx.x]);
    };
    auto keep_requested = [&](uint32_t b) {
        if (threadIdx.x < p.K) { pos_of[b][threadIdx.x] = next_pos; weight_of[b][threadIdx.x] = next_weight; }
    };
    // (the routing is from before the kernel in front)
    request(blockIdx.x);
    keep_requested(0);
    pdl_wait();
    pdl_launch_dependents();
    __syncthreads();
    for (uint32_t tok = blockIdx.x, buf = 0; tok < p.tokens; tok += gridDim.x, buf ^= 1u) {
        const uint32_t *pos = pos_of[buf];
        const float *wk = weight_of[buf];
        const bool more = tok + gridDim.x < p.tokens;
        if (more) request(tok + gridDim.x);
        const float gate = p.gate_val != nullptr ? p.gate_val[tok] : 0.0f;
        for (uint32_t d = threadIdx.x * 8u; d < p.D; d += 2048u) {
            const size_t i = (size_t)tok * p.D + d;
            Part8<PART> v[kMaxTopK];
#pragma unroll
            for (uint32_t r = 0; r < (uint32_t)kMaxTopK; ++r)
                if (r < p.K && pos[r] != kBpNotLocal) v[r].load(p.partial, (size_t)pos[r] * p.D + d);
            if (p.partial_y != nullptr) {          // expert parallelism: this rank's share of the sum
                float acc[8] = {};
#pragma unroll
                for (uint32_t r = 0; r < (uint32_t)kMaxTopK; ++r)
                    if (r < p.K && pos[r] != kBpNotLocal)
#pragma unroll
                        for (int k = 0; k < 8; ++k) acc[k] += wk[r] * v[r].at(k);
                store_out8<OUT_F32>(p.partial_y, i, acc, p.aligned);
                continue;
            }
            float y[8], hid[8] = {}, delta[8] = {};
            if (p.hidden != nullptr) load_out8<OUT>(p.hidden, i, hid, p.aligned);
            if (p.hidden_delta != nullptr) load_out8<OUT_F16>(p.hidden_delta, i, delta, p.aligned);
            float h1[8] = {};
            if (p.shared_partial != nullptr) {
                if (p.shared_half) load_out8<OUT_F16>(p.shared_partial, i, h1); else load_out8<OUT_F32>(p.shared_partial, i, h1);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    h1[k] = round_out<OUT>(h1[k]);
                    if (p.gate_val != nullptr) h1[k] = round_out<OUT>(sigmoid_div(h1[k], gate));
                }
            }
            if (p.prefill) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    float h2 = 0.0f;
#pragma unroll
                    for (uint32_t r = 0; r < (uint32_t)kMaxTopK; ++r)
                        if (r < p.K) h2 = fmaf(wk[r], round_out<OUT>(v[r].at(k)), h2);
                    h2 = round_out<OUT>(h2);
                    y[k] = h1[k] + h2;
                    hid[k] = round_out<OUT>(hid[k] + h1[k]) + h2;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    float acc = h1[k];
#pragma unroll
                    for (uint32_t r = 0; r < (uint32_t)kMaxTopK; ++r)
                        if (r < p.K) acc += wk[r] * v[r].at(k);
                    y[k] = round_out<OUT>(acc);
                    if (p.hidden_delta != nullptr) hid[k] = round_out<OUT>(hid[k] + delta[k]);
                    hid[k] += y[k];
                }
            }
            if (p.y != nullptr) store_out8<OUT>(p.y, i, y, p.aligned);
            if (p.hidden != nullptr) store_out8<OUT>(p.hidden, i, hid, p.aligned);
            if constexpr (NORM)
#pragma unroll
                for (int k = 0; k < 8; ++k) row[d + k] = y[k];
        }
        if (more) keep_requested(buf ^ 1u);
        if constexpr (NORM) {
            // the reduction tree of stage_x (staged_decode.cuh), so that a stack's rows have the bits of its layers run one by one
            __syncthreads();
            float keep[kBpNormRow / 256], ss = 0.0f;
#pragma unroll
            for (uint32_t j = 0; j < kBpNormRow / 256; ++j) {
                const uint32_t i = threadIdx.x + j * 256u;
                keep[j] = i < p.D ? row[i] : 0.0f;
            }
#pragma unroll
            for (uint32_t j = 0; j < kBpNormRow / 256; ++j) ss = fmaf(keep[j], keep[j], ss);
            ss = warp_sum(ss);
            if ((threadIdx.x & 31u) == 0) wsum[threadIdx.x >> 5] = ss;
            __syncthreads();
            float tot = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) tot += wsum[i];
            const float sc = rsqrtf(tot / (float)p.D + 1e-6f);
#pragma unroll
            for (uint32_t j = 0; j < kBpNormRow / 256; ++j) {
                const uint32_t i = threadIdx.x + j * 256u;
                if (i < p.D) p.x_next[(size_t)tok * p.D + i] = __float2half_rn(keep[j] * sc);
            }
        }
        __syncthreads();
    }
}

}  // namespace nvmai
