// Few rows per expert: the weights streamed once through the warps' own tensor-core steps (mma.sync on the codes).
//
// With up to 16 rows per expert the conversion of the codes to fp16 operands is what the grouped GEMMs of
// expert_gemm.cuh spend their time on (154 issue slots per 1,024 codes in gate/up, everything included).  mma.sync takes the codes as they are
// (tile_gemv.cuh: a code in the low mantissa bits of a half is an exact subnormal) and applies scale and bias once per
// group in fp32: 75 slots per 1,024 8-bit codes for 8 rows, everything included, and nothing is rounded.  Every row's result has
// the bits of the single-row stages: the fp32 chains of the parts of a row (an eighth of the groups each in gate/up, a
// half in down) and their sum run in the same order (gate_up_compute, down_warp in staged_decode.cuh).
//
// One block per SM, 16 compute warps and one that issues the copies.  A unit = an item (an expert, up to 8 * NB of its
// rows as tensor-core columns) x 64 or 128 features (phase 0: gate and up rows of each) or 256 rows of the down
// projection (phase 1); a block takes consecutive units, so the rows of an item are staged once for several of them.
// The codes come as boxes of 64 rows x 128 bytes, 32 KB a stage, as many stages (two to six) as the shared memory holds.  KS = 2: two warps
// share a tile, each half of K, so that a unit is small enough to balance over the chip.  96 registers a thread are what 18
// warps leave; two column blocks (NB = 2) spill 28 to 200 bytes of them.
#pragma once

#include "batch_path.h"
#include "decode_kernels.cuh"
#include "tcgen05.cuh"

namespace nvmai {

constexpr int kSgWarps = 16;
constexpr int kSgThreads = (kSgWarps + 1) * 32;
constexpr uint32_t kSgBoxBytes = 64 * 128, kSgStageBytes = 4 * kSgBoxBytes;
constexpr uint32_t kSgMaxStages = 6;

struct SgBarriers {
    uint64_t full[kSgMaxStages], empty[kSgMaxStages];
    uint64_t m_full[2], m_empty[2];
    uint64_t x_full, x_empty, x_ready;      // rows landed; free again; in fragment order
    uint64_t h_full[2][8];                  // KS = 2: a tile's first half handed over
};
static_assert(kSgWarps == 16, "wide rows: a row per warp");
static_assert(sizeof(SgBarriers) <= 1024, "the barriers have 1 KB");

struct SgUnit { uint32_t item, shared, expert, start, count, j; };
__device__ __forceinline__ SgUnit sg_unit(const SgParams &p, uint32_t u) {
    SgUnit r;
    r.item = u / p.units_per_item;
    r.j = u - r.item * p.units_per_item;
    r.shared = r.item < p.shared_items ? 1u : 0u;
    if (r.shared) {
        r.expert = 0;
        r.start = r.item * p.cap;
        r.count = min(p.cap, p.tokens - r.start);
    } else {
        const WorkItem w = p.work[r.item - p.shared_items];
        r.expert = min(w.expert, p.num_experts - 1u);
        r.start = w.start;
        r.count = min(w.count, p.cap);
    }
    return r;
}

// 8 halves in memory order -> the order of the B fragments (permute_x in tile_gemv.cuh)
template <int BITS> __device__ __forceinline__ uint4 sg_permute8(const uint4 &q) {
    if (BITS == 4) return make_uint4(__byte_perm(q.x, q.z, 0x5410), __byte_perm(q.x, q.z, 0x7632),
                                     __byte_perm(q.y, q.w, 0x5410), __byte_perm(q.y, q.w, 0x7632));
    return make_uint4(__byte_perm(q.x, q.y, 0x5410), __byte_perm(q.x, q.y, 0x7632),
                      __byte_perm(q.z, q.w, 0x5410), __byte_perm(q.z, q.w, 0x7632));
}

template <int BITS> struct SgCodes;
template <> struct SgCodes<4> { using vec = uint2; };
template <> struct SgCodes<8> { using vec = uint4; };
__device__ __forceinline__ void sg_lds(uint2 &v, uint32_t a) { asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a)); }
__device__ __forceinline__ void sg_lds(uint4 &v, uint32_t a) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
}
__device__ __forceinline__ void sg_lds(uint32_t &v, uint32_t a) { asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); }
__device__ __forceinline__ uint32_t sg_lds16(uint32_t a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float sg_lds_f32(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

// One group of a 16-row tile against 8 NB columns: the arithmetic of group_step.
template <int BITS, int META, int NB>
__device__ __forceinline__ void sg_group(uint32_t code_a, uint32_t code_b, uint32_t x_at, uint32_t x_block, uint16_t sa, uint16_t sb,
                                         uint16_t ba, uint16_t bb, const float (&xs)[NB][2], float (&acc)[NB][4]) {
    typename SgCodes<BITS>::vec va, vb;
    sg_lds(va, code_a);
    sg_lds(vb, code_b);
    uint32_t pa[8], pb[8];
    unpack_group<BITS>(va, pa);
    unpack_group<BITS>(vb, pb);
    const float fsa = meta_to_float<META>(sa) * kCodeUnscale, fsb = meta_to_float<META>(sb) * kCodeUnscale;
    const float fba = meta_to_float<META>(ba), fbb = meta_to_float<META>(bb);
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        uint4 lo, hi;
        sg_lds(lo, x_at + n * x_block);
        sg_lds(hi, x_at + n * x_block + 16u);
        const uint32_t xb[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < 4; ++s)
            mma16816(d, pa[2 * s], pb[2 * s], pa[2 * s + 1], pb[2 * s + 1], xb[2 * s], xb[2 * s + 1]);
        acc[n][0] = fmaf(fsa, d[0], acc[n][0]); acc[n][0] = fmaf(fba, xs[n][0], acc[n][0]);
        acc[n][2] = fmaf(fsb, d[2], acc[n][2]); acc[n][2] = fmaf(fbb, xs[n][0], acc[n][2]);
        acc[n][1] = fmaf(fsa, d[1], acc[n][1]); acc[n][1] = fmaf(fba, xs[n][1], acc[n][1]);
        acc[n][3] = fmaf(fsb, d[3], acc[n][3]); acc[n][3] = fmaf(fbb, xs[n][1], acc[n][3]);
    }
}

// BITS, META: codes and scales; OUT: type of the activations; PHASE 0 gate/up, 1 down; NB: column blocks of 8 rows.
// QUADS 1, 2: the parts of a row are whole quads of groups (sg_quads: a multiple of 2048 inputs in phase 0, where KS = 2
// then, of 512 in phase 1), so scales, biases and row sums are read four at a time; 1: a part is one quad, its code
// without the loop (with it, 4 rows of 2048 / 512 took 49.2 us instead of 48.4, 13 rows 66.2 instead of 64.8); 2: any
// number of quads; 0: other shapes.
template <int BITS, int META, int OUT, int PHASE, int NB, int QUADS>
__global__ void __launch_bounds__(kSgThreads + 32, 1) stream_gemm_kernel(const __grid_constant__ SgArgs args) {
    const SgParams &p = args.p;
    constexpr uint32_t KS = PHASE == 0 && QUADS != 0 ? 2u : 1u;
    constexpr uint32_t kChunkGroups = BITS == 4 ? 4u : 2u;        // groups in 128 bytes of a row
    constexpr uint32_t kRows = PHASE == 0 ? 128u / KS : 256u;     // features (phase 0) or down rows of a unit
    constexpr uint32_t kCols = 8u * NB;
    constexpr bool kWideRows = PHASE == 1 && OUT == OUT_F32;      // activation rows come as fp32
    extern __shared__ unsigned char sg_smem_raw[];
    const uint32_t raw = smem_addr(sg_smem_raw), base = (raw + 1023u) & ~1023u;
    unsigned char *gen = sg_smem_raw + (base - raw);
    SgBarriers *bars = reinterpret_cast<SgBarriers *>(gen);
    const uint32_t ring = base + 1024u, meta0 = base + p.meta_off, xbuf = base + p.x_off;
    const uint32_t groups = p.kdim / 64u, row_stride = p.kdim * 2u + 16u, sum_stride = groups + 4u;
    float *xsum = reinterpret_cast<float *>(gen + p.sum_off);                  // [kCols][sum_stride]
    float *scale_up = reinterpret_cast<float *>(gen + p.scale_off);            // [kCols]
    float *handover = scale_up + kCols;                                        // KS = 2: [2][8 tiles][4 NB][32]
    const uint32_t meta_bytes = kRows * groups * 2u;                           // one matrix's scales (or biases) of a unit
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

    if (tid == 0) {
        for (uint32_t i = 0; i < kSgMaxStages; ++i) { mbar_init(&bars->full[i], 1); mbar_init(&bars->empty[i], kSgWarps); }
        for (uint32_t i = 0; i < 2; ++i) { mbar_init(&bars->m_full[i], 1); mbar_init(&bars->m_empty[i], kSgWarps); }
        mbar_init(&bars->x_full, 1); mbar_init(&bars->x_empty, kSgWarps); mbar_init(&bars->x_ready, kSgWarps);
        for (uint32_t i = 0; i < 16; ++i) mbar_init(&bars->h_full[i >> 3][i & 7], 1);
        mbar_fence_init();
    }
    // Codes, scales and the work list do not come from the kernel in front (list_ready): the warp that requests them then does
    // so without waiting for it, and only those that touch rows wait.  As much of a block's weights as the ring holds (up to
    // 192 KB) is on its way while the slowest block of the kernel in front still runs and while its writes are flushed.
    auto wait_in_front = [&]() {
        pdl_wait();
        pdl_launch_dependents();
    };
    if (!p.beside && !p.list_ready) wait_in_front();
    const bool late_wait = !p.beside && p.list_ready;
    bool ok = __syncthreads_and(*reinterpret_cast<volatile unsigned int *>(p.status) == 0u);
    // the units of the launch: those of the shared items come first and are skipped where another kernel has them
    const uint32_t skip = *p.shared_on != 0u ? 0u : p.shared_items * p.units_per_item;
    const uint32_t total = ok ? (p.shared_items + p.n_work[0]) * p.units_per_item - skip : 0u;
    const uint32_t u0 = skip + (uint32_t)((unsigned long long)total * blockIdx.x / gridDim.x);
    const uint32_t u1 = skip + (uint32_t)((unsigned long long)total * (blockIdx.x + 1) / gridDim.x);
    const uint32_t n_chunk = (p.kdim * BITS / 8u + 127u) / 128u / KS;          // stages of a unit
    constexpr uint32_t kMats = PHASE == 0 ? 2u : 1u;

    if (warp == kSgWarps) {
        // ---------------- codes, scales, biases ----------------
        if (elect_one()) {
            uint32_t s = 0, s_ph = 0, mb = 0, m_ph = 0;
            for (uint32_t u = u0; u < u1 && ok; ++u) {
                const SgUnit un = sg_unit(p, u);
                const uint8_t *blob = p.experts + (size_t)un.expert * p.stride;
                const uint32_t row0 = un.j * kRows;
                ok = mbar_wait(&bars->m_empty[mb], m_ph ^ 1u, p.status);
                if (!ok) break;
                mbar_expect_tx(&bars->m_full[mb], 2u * kMats * meta_bytes);
                unsigned char *dst = gen + p.meta_off + mb * p.meta_bytes;
#pragma unroll
                for (uint32_t m = 0; m < kMats; ++m) {
                    const size_t at = (size_t)row0 * groups * 2u;
                    bulk_g2s(dst + m * meta_bytes, (un.shared ? p.shared_s[m] : blob + p.off_s[m]) + at, meta_bytes, &bars->m_full[mb]);
                    bulk_g2s(dst + (kMats + m) * meta_bytes, (un.shared ? p.shared_b[m] : blob + p.off_b[m]) + at, meta_bytes, &bars->m_full[mb]);
                }
                if ((mb ^= 1u) == 0u) m_ph ^= 1u;
                const CUtensorMap *map0 = un.shared ? &args.shared0 : &args.routed0, *map1 = un.shared ? &args.shared1 : &args.routed1;
                for (uint32_t i = 0; i < n_chunk; ++i) {
                    ok = mbar_wait(&bars->empty[s], s_ph ^ 1u, p.status);
                    if (!ok) break;
                    mbar_expect_tx(&bars->full[s], kSgStageBytes);
                    const uint32_t at = ring + s * kSgStageBytes;
#pragma unroll
                    for (uint32_t b = 0; b < 4u; ++b) {
                        // KS = 2: gate, up of the first half of K, then of the second; else the rows of gate, then up / down
                        const uint32_t k = i * 128u + (KS == 2u ? (b >> 1) * (n_chunk * 128u) : 0u);
                        const CUtensorMap *map = PHASE == 0 && (KS == 2u ? (b & 1u) : (b >> 1)) ? map1 : map0;
                        const uint32_t r = row0 + (PHASE == 1 ? b * 64u : KS == 2u ? 0u : (b & 1u) * 64u);
                        tma_load_3d(at + b * kSgBoxBytes, map, k, r, un.expert, &bars->full[s]);
                    }
                    if (++s == p.stages) { s = 0; s_ph ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else if (warp == kSgWarps + 1) {
        // ---------------- rows of an item ----------------
        if (late_wait) wait_in_front();
        uint32_t ph = 0;
        const uint32_t bytes = p.kdim * (kWideRows ? 4u : 2u);
        for (uint32_t u = u0; u < u1 && ok; u = (u / p.units_per_item + 1u) * p.units_per_item) {
            const SgUnit un = sg_unit(p, u);
            const uint8_t *src = static_cast<const uint8_t *>(un.shared ? p.shared_rows : p.rows);
            size_t row = 0;
            if ((uint32_t)lane < un.count) {
                row = un.start + lane;
                if (PHASE == 0 && !un.shared) row = p.sorted_pair[row] / p.top_k;
            }
            ok = __all_sync(0xffffffffu, mbar_wait(&bars->x_empty, ph ^ 1u, p.status));
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(&bars->x_full, un.count * bytes);
            __syncwarp();
            if ((uint32_t)lane < un.count)
                bulk_g2s(gen + (kWideRows ? p.raw_off + lane * bytes : p.x_off + lane * row_stride), src + row * bytes, bytes, &bars->x_full);
            ph ^= 1u;
        }
    } else {
        // ---------------- compute ----------------
        if (late_wait) wait_in_front();
        const uint32_t g = lane >> 2, t = lane & 3u;
        const uint32_t ks = KS == 2u ? warp >> 3 : 0u, tl = KS == 2u ? warp & 7u : warp;
        // the lane's rows: phase 0 gate and up of feature 8 tl + g, phase 1 rows 16 tl + g and + 8
        const uint32_t box_a = PHASE == 1 ? tl >> 2 : KS == 2u ? 2u * ks : tl >> 3;
        const uint32_t box_b = PHASE == 1 ? box_a : KS == 2u ? box_a + 1u : box_a + 2u;
        const uint32_t r_a = (PHASE == 1 ? (tl & 3u) * 16u : (tl & 7u) * 8u) + g, r_b = PHASE == 1 ? r_a + 8u : r_a;
        const uint32_t in_row = BITS == 4 ? ((((t >> 1) ^ g) << 4) | ((t & 1u) << 3)) : ((t ^ g) << 4);
        const uint32_t code_a = ring + box_a * kSgBoxBytes + r_a * 128u + in_row, code_b = ring + box_b * kSgBoxBytes + r_b * 128u + in_row;
        const uint32_t m_row = PHASE == 1 ? tl * 16u + g : tl * 8u + g;
        const uint32_t m_a = m_row * groups * 2u, m_b = PHASE == 1 ? m_a + 8u * groups * 2u : m_a + meta_bytes;
        const uint32_t x_at = xbuf + g * row_stride + t * 32u, x_block = 8u * row_stride;
        uint32_t s = 0, s_ph = 0, mb = 0, m_ph = 0, x_ph = 0, item = 0xFFFFFFFFu, turn = 0;
        SgUnit next = u0 < u1 ? sg_unit(p, u0) : SgUnit{};
        for (uint32_t u = u0; u < u1; ++u) {
            const SgUnit un = next;
            if (u + 1u < u1) next = sg_unit(p, u + 1u);
            if (un.item != item) {
                // the item's rows: into fragment order, with the sums of their groups (8 lanes a group)
                item = un.item;
                ok = __all_sync(0xffffffffu, mbar_wait(&bars->x_full, x_ph, p.status));
                x_ph ^= 1u;
                if (ok && kWideRows) {
                    // fp32 rows: scaled by a power of two into fp16's range first (stage_row_part)
                    for (uint32_t r = warp; r < un.count; r += kSgWarps) {
                        const float *src = reinterpret_cast<const float *>(gen + p.raw_off) + r * p.kdim;
                        float m = 0.0f;
                        for (uint32_t i = lane * 4u; i < p.kdim; i += 128u) {
                            const float4 v = *reinterpret_cast<const float4 *>(src + i);
                            m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
                        }
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                        const uint32_t ebits = (__float_as_uint(m) >> 23) & 0xFFu;
                        const bool big = ebits > 14u;
                        const float down = big ? __uint_as_float((268u - ebits) << 23) : 1.0f;
                        if (lane == 0) scale_up[r] = big ? __uint_as_float((ebits - 14u) << 23) : 1.0f;
                        for (uint32_t i = lane * 4u; i < p.kdim; i += 128u) {
                            const float4 v = *reinterpret_cast<const float4 *>(src + i);
                            const __half2 lo = __floats2half2_rn(v.x * down, v.y * down), hi = __floats2half2_rn(v.z * down, v.w * down);
                            *reinterpret_cast<uint2 *>(gen + p.x_off + r * row_stride + i * 2u) =
                                make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
                        }
                    }
                }
                // wide rows: the warp goes on with the rows it has just written; else the groups of all rows over all warps
                const uint32_t n_all = un.count * groups;
                uint32_t first = kWideRows ? warp * groups : warp * 4u;
                const uint32_t step = kWideRows ? 4u : kSgWarps * 4u;
                __syncwarp();
                for (uint32_t end = kWideRows ? min(first + groups, n_all) : n_all; ok && first < end; first += step) {
                    const uint32_t id = first + (lane >> 3), r = id / groups, G = id - r * groups;
                    const bool live = id < end;
                    uint4 *at = reinterpret_cast<uint4 *>(gen + p.x_off + r * row_stride + G * 128u + (lane & 7u) * 16u);
                    float v = 0.0f;
                    if (live) {
                        const uint4 q = *at;
                        const __half2 *h = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
                        for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); v += f.x; v += f.y; }
                        *at = sg_permute8<BITS>(q);
                    }
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                    v += __shfl_xor_sync(0xffffffffu, v, 4);
                    if (live && (lane & 7) == 0) xsum[r * sum_stride + G] = v;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->x_ready);
                ok = __all_sync(0xffffffffu, mbar_wait(&bars->x_ready, x_ph ^ 1u, p.status) && ok);
                if (!ok) break;
            }
            ok = __all_sync(0xffffffffu, mbar_wait(&bars->m_full[mb], m_ph, p.status) && ok);
            if (!ok) break;
            const uint32_t meta = meta0 + mb * p.meta_bytes;
            const uint32_t bias = meta + kMats * meta_bytes;
            float tot[NB][4] = {}, part[QUADS != 0 && PHASE == 0 ? 4 : 1][NB][4];
            float su[NB][2];
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                su[n][0] = kWideRows ? scale_up[n * 8u + 2u * t] : 1.0f;
                su[n][1] = kWideRows ? scale_up[n * 8u + 2u * t + 1u] : 1.0f;
            }
            auto stage_wait = [&]() { ok = __all_sync(0xffffffffu, mbar_wait(&bars->full[s], s_ph, p.status)); };
            auto stage_done = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->empty[s]);
                if (++s == p.stages) { s = 0; s_ph ^= 1u; }
            };
            if (QUADS != 0) {
                constexpr uint32_t kParts = PHASE == 0 ? 4u : 2u;
                auto quad = [&](uint32_t G0, float (&acc)[NB][4]) {
                    uint2 sa, sb, ba, bb;                 // the quad's scales and biases of both rows
                    sg_lds(sa, meta + m_a + G0 * 2u); sg_lds(sb, meta + m_b + G0 * 2u);
                    sg_lds(ba, bias + m_a + G0 * 2u); sg_lds(bb, bias + m_b + G0 * 2u);
                    float xs[4][NB][2];
#pragma unroll
                    for (int n = 0; n < NB; ++n)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const float4 v = *reinterpret_cast<const float4 *>(xsum + (n * 8u + 2u * t + c) * sum_stride + G0);
                            xs[0][n][c] = v.x; xs[1][n][c] = v.y; xs[2][n][c] = v.z; xs[3][n][c] = v.w;
                        }
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j) {
                        if (j % kChunkGroups == 0u) { stage_wait(); if (!ok) break; }
                        const uint32_t at = s * kSgStageBytes, jx = (j % kChunkGroups) * (BITS == 4 ? 32u : 64u);
                        sg_group<BITS, META, NB>((code_a + at) ^ jx, (code_b + at) ^ jx, x_at + (G0 + j) * 128u, x_block, meta_pick(sa, j),
                                                 meta_pick(sb, j), meta_pick(ba, j), meta_pick(bb, j), xs[j], acc);
                        if (j % kChunkGroups == kChunkGroups - 1u) stage_done();
                    }
                };
                const uint32_t part_groups = groups / (PHASE == 0 ? 8u : 2u);
#pragma unroll
                for (uint32_t q = 0; q < kParts; ++q) {
                    float acc[NB][4] = {};
                    if constexpr (QUADS == 1) {
                        quad((ks * kParts + q) * 4u, acc);
                    } else {
                        const uint32_t G1 = (ks * kParts + q + 1u) * part_groups;
                        for (uint32_t G0 = G1 - part_groups; ok && G0 < G1; G0 += 4u) quad(G0, acc);
                    }
                    if (!ok) break;
#pragma unroll
                    for (int n = 0; n < NB; ++n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if (PHASE == 0) part[q][n][i] = acc[n][i];
                            else tot[n][i] += acc[n][i] * su[n][i & 1];
                        }
                }
            } else {
                // any shape: parts of ceil(groups / 8) groups (gate/up) or ceil(groups / 2) (down), one group at a time
                const uint32_t gpp = PHASE == 0 ? (groups + 7u) / 8u : (groups + 1u) / 2u;
                float acc[NB][4] = {};
                for (uint32_t G = 0; G < groups; ++G) {
                    if (G % kChunkGroups == 0u) { stage_wait(); if (!ok) break; }
                    const uint32_t at = s * kSgStageBytes, jx = (G % kChunkGroups) * (BITS == 4 ? 32u : 64u);
                    float xs[NB][2];
#pragma unroll
                    for (int n = 0; n < NB; ++n) {
                        xs[n][0] = xsum[(n * 8u + 2u * t) * sum_stride + G];
                        xs[n][1] = xsum[(n * 8u + 2u * t + 1u) * sum_stride + G];
                    }
                    sg_group<BITS, META, NB>((code_a + at) ^ jx, (code_b + at) ^ jx, x_at + G * 128u, x_block, (uint16_t)sg_lds16(meta + m_a + G * 2u),
                                             (uint16_t)sg_lds16(meta + m_b + G * 2u), (uint16_t)sg_lds16(bias + m_a + G * 2u),
                                             (uint16_t)sg_lds16(bias + m_b + G * 2u), xs, acc);
                    if ((G + 1u) % gpp == 0u || G + 1u == groups) {
#pragma unroll
                        for (int n = 0; n < NB; ++n)
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                tot[n][i] += PHASE == 0 ? acc[n][i] : acc[n][i] * su[n][i & 1];
                                acc[n][i] = 0.0f;
                            }
                    }
                    if ((G + 1u) % kChunkGroups == 0u || G + 1u == groups) stage_done();
                }
            }
            if (!ok) break;
            // with its last unit the item's rows are done with
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && (u + 1u == u1 || next.item != item)) mbar_arrive(&bars->x_empty);
            // The unit's scales too, but with KS = 2 only once the hand-over below has been read: the scales of the unit
            // after the next come when every warp has released these, and the first half's warp needs them before it
            // writes this hand-over slot again.  (The ring of codes would hold that warp back as well, but only while its
            // stages are fewer than two units'.)
            auto scales_done = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->m_empty[mb]);
                if ((mb ^= 1u) == 0u) m_ph ^= 1u;
            };
            if (KS == 1u) scales_done();
            if (PHASE == 0) {
                bool mine = true;
                if (QUADS != 0) {
                    // the first half's running sum goes to the warp of the second half, which goes on from there
                    float *h = handover + (((turn & 1u) * 8u + tl) * (4u * NB)) * 32u + lane;
                    if (ks == 0u) {
#pragma unroll
                        for (int n = 0; n < NB; ++n)
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                h[(n * 4 + i) * 32] = (((0.0f + part[0][n][i]) + part[1][n][i]) + part[2][n][i]) + part[3][n][i];
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars->h_full[turn & 1u][tl]);
                        mine = false;
                    } else {
                        ok = __all_sync(0xffffffffu, mbar_wait(&bars->h_full[turn & 1u][tl], (turn >> 1) & 1u, p.status));
                        if (!ok) break;
#pragma unroll
                        for (int n = 0; n < NB; ++n)
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                tot[n][i] = (((h[(n * 4 + i) * 32] + part[0][n][i]) + part[1][n][i]) + part[2][n][i]) + part[3][n][i];
                    }
                    scales_done();
                    ++turn;
                }
                if (mine) {
                    const uint32_t f = un.j * kRows + tl * 8u + g;
                    void *out = un.shared ? p.shared_out : p.out;
#pragma unroll
                    for (int n = 0; n < NB; ++n)
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            const uint32_t col = n * 8u + 2u * t + c;
                            if (col < un.count) {
                                float gate = tot[n][c], up = tot[n][2 + c];
                                if (un.shared) { gate = round_mid<OUT>(gate); up = round_mid<OUT>(up); }
                                store_mid<OUT>(out, (size_t)(un.start + col) * p.out_cols + f, hidden_act(gate, p.act) * up);
                            }
                        }
                }
            } else {
                const uint32_t d = un.j * kRows + tl * 16u + g;
                float *out = static_cast<float *>(un.shared ? p.shared_out : p.out);
#pragma unroll
                for (int n = 0; n < NB; ++n)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const uint32_t col = n * 8u + 2u * t + c;
                        if (col < un.count) {
                            float *o = out + (size_t)(un.start + col) * p.out_cols + d;
                            o[0] = tot[n][c];
                            o[8] = tot[n][2 + c];
                        }
                    }
            }
        }
    }
    __syncwarp();
    if (!__syncthreads_and(ok)) {          // given up: let the copies in flight land before the memory is released
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    if (p.beside) {                        // the kernel after this one relies on the one before it being complete
        pdl_wait();
        pdl_launch_dependents();
    }
}

}  // namespace nvmai
