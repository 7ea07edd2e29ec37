// Batched experts as grouped GEMMs on the 5th-generation tensor cores: the routed and shared experts of a prefill
// chunk or of a decode batch.
//
// What it replaces: prefill_grouped_routed_moe_batched_phase1/_down (prefill.metal:460-534), which evaluate every
// (pair, feature) dot product on its own with no reuse of an expert's weights across its tokens, and
// PrefillSharedExpert.encodeBlock (PrefillSharedExpert.swift:13-60), which repeats the decode GEMVs per token row.
//
// D[128 x N] (+)= A[128 x 16] * B[N x 16]^T per instruction: 128 weight rows are the M operand, the N token rows of a
// work item (an expert and up to `cap` of the rows routed to it, consecutive in sorted pair order) the N operand, so a
// short item costs a narrow instruction instead of a padded tile.
//   phase 0: gate and up tiles of the same 128 features side by side; epilogue act(gate) * up
//   phase 1: tiles of 128 rows of the down projection one after another, the item's activation rows staying in shared
//            memory for all tiles of a unit; epilogue -> partial[row][d]
//
// One block per SM runs for the whole launch and walks the units (item x feature tile, item x run of down tiles).
// Roles (31 warps):
//   16 producer warps  codes -> fp16 A tiles in TENSOR memory (tcgen05.st), four groups of four warps, each group every
//                      fourth A stage (128 rows x 64 K values)
//   8 epilogue warps   accumulators -> activations / partial rows, while the next unit's MMAs run
//   4 warps for the token rows, 2 threads that issue MMAs (phase 0: one per tile; phase 1: one), 1 warp for the TMA loads of
//   the packed codes and scales
//
// Where an item leaves room for one set of accumulators only (more than 96 rows), the MMAs wait until the epilogue has emptied
// them and the producers have nothing to convert for, so all 24 warps empty them.
//
// Why A goes through tensor memory: with both operands in shared memory an MMA of N <= 128 columns is bound by reading
// the 4 KB of A per instruction (measured 39 cycles at N = 16, 48 at N = 64, 64 at N = 128, and the producers' stores
// compete for the same bandwidth); with A in tensor memory the same instruction takes N / 2 cycles (9 at N = 16).
//
// Operand exactness: the tensor core multiplies the CENTRED weight s * (q - c), c = 8; a bf16 scale has 8 significant
// bits and |q - 8| <= 8, so the product is exact in fp16.  An 8-bit code goes through as its two nibbles,
// 16 s * (hq - 8) and s * (lq - 8), two stages against the same B rows.  An fp16 scale (11 bits) is rounded once
// (kSplit = false, the prefill path) or goes through as two scales of 8 and 3 bits (kSplit = true, exact; the decode
// path).  The rest of w = q*s + b, the per-group constant b + c*s, enters through extra K blocks: every B row carries
// the sums of its groups (fp16 hi + lo) and the producers append the constants as [hi | hi | lo] columns against
// [X_hi | X_lo | X_hi].  Phase 1 rows carry sums of half groups (32 values): that is what one epilogue warp holds.
//
// Every wait is bounded; on expiry the status word is set, the block waits for its copies in flight, frees its tensor
// memory and returns, and blocks that start later return at once.
#pragma once

#include "batch_path.h"
#include "decode_kernels.cuh"
#include "tcgen05.cuh"

namespace nvmai {

constexpr int kEgProducerWarps = 16, kEgEpilogueWarps = 8, kEgRowWarps = 4;
constexpr int kEgRowWarp0 = 24, kEgMmaWarp = 28, kEgCodeWarp = 29, kEgMmaWarp1 = 30;
constexpr int kEgThreads = 31 * 32;
// Tensor memory: accumulators from column 0 on, A slots (two stages of 128 rows x 64 fp16 each) at the end.
constexpr uint32_t kEgMaxPairs = 6;
constexpr uint32_t kEgCols = 512, kEgStageCols = 32, kEgSlotCols = 2 * kEgStageCols;
constexpr uint32_t kEgChunkBytes = 128 * 128; // codes of 128 rows: 128 bytes of each
constexpr uint32_t kEgMaxRowSlots = 16, kEgMaxMeta = 4, kEgMaxAcc = 8;

struct EgBarriers {
    uint64_t a_full[kEgMaxPairs][2], a_empty[kEgMaxPairs][2];      // phase 0: per tile; phase 1: [.][0]
    uint64_t c_full[kEgChunks], c_empty[kEgChunks];
    uint64_t m_full[kEgMaxMeta], m_empty[kEgMaxMeta];
    uint64_t b_full[kEgMaxRowSlots], b_empty[kEgMaxRowSlots];
    uint64_t d_full[kEgMaxAcc], d_empty[kEgMaxAcc];
    uint32_t tmem_slot;
};
static_assert(sizeof(EgBarriers) <= 1024, "the barriers have 1 KB");

// One unit of the launch.
struct EgUnit { uint32_t shared, expert, start, count, j; };

__device__ __forceinline__ EgUnit eg_unit(const EgParams &p, uint32_t u, uint32_t shared_items) {
    EgUnit r;
    const uint32_t item = u / p.units_per_item;
    r.j = u - item * p.units_per_item;
    r.shared = item < shared_items ? 1u : 0u;
    if (r.shared) {       // the shared expert sees every token: even runs of token rows, first because they are the longest
        const uint32_t even = p.tokens / p.shared_items, extra = p.tokens - even * p.shared_items;
        r.expert = 0;
        r.start = item * even + min(item, extra);
        r.count = even + (item < extra ? 1u : 0u);
    } else {
        const WorkItem w = p.work[item - shared_items];
        r.expert = min(w.expert, p.num_experts - 1u);
        r.start = w.start;
        r.count = min(w.count, p.cap);
    }
    return r;
}

// For roles that must not wait for the work list between two units: the next unit is requested a unit ahead.
__device__ __forceinline__ EgUnit eg_unit_or_last(const EgParams &p, uint32_t u, uint32_t total, uint32_t shared_items) {
    if (total == 0u) return EgUnit{};
    return eg_unit(p, min(u, total - 1u), shared_items);
}

// The scale a stage multiplies by, twice in a register: the low (odd = 0) or high half of `word`, pass 0 .. PASSES-1 =
// (8-bit: high nibble, low nibble) x (SPLIT: the 8 leading significant bits of an fp16 scale, the rest).
template <int BITS, int META, bool SPLIT>
__device__ __forceinline__ __half2 eg_pass_scale(uint32_t word, uint32_t odd, uint32_t pass) {
    uint32_t s;
    if (META == META_FP16) {
        s = __byte_perm(word, word, odd ? 0x3232 : 0x1010);
    } else {
        const float f = __uint_as_float(__byte_perm(word, 0u, odd ? 0x3244 : 0x1044));
        const __half2 h = __floats2half2_rn(f, f);
        s = *reinterpret_cast<const uint32_t *>(&h);
    }
    __half2 r = *reinterpret_cast<const __half2 *>(&s);
    if (SPLIT) {
        const uint32_t lead = s & 0xFFF8FFF8u;
        const __half2 hi = *reinterpret_cast<const __half2 *>(&lead);
        r = (pass & 1u) ? __hsub2(r, hi) : hi;
        pass >>= 1;
    }
    if (BITS == 8 && pass == 0u) r = __hmul2(r, __float2half2_rn(16.0f));
    return r;
}

// 64 codes of one row -> 32 registers of fp16 pairs, in the K order bp_k_order (4-bit) or the natural one (8-bit).
// The logic pipe runs at half rate and bounds the conversion, so the work goes to the fp16 arithmetic where it can:
// a byte b = lo + 16 hi of the word becomes 1024 + b (one byte permute for two bytes) and, with the low nibble masked
// off, 1024 + 16 hi; their difference is lo exactly, fma(lo, s, -8 s) = s * (lo - 8) rounds once and is exact, and
// hi comes as (16 (hi - 8)) * (s / 16), exact unless s / 16 is an fp16 subnormal.  SPLIT scales can be that small:
// there the high nibble is scaled down first (16 (hi - 8) / 16).
template <bool SPLIT>
__device__ __forceinline__ void eg_convert4(const uint4 &a, const uint4 &b, __half2 s2, uint32_t (&o)[32]) {
    const __half2 k_hi = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));     // 1024 + 128
    const __half2 sixteenth = __float2half2_rn(0.0625f);
    const __half2 s16 = __hmul2(s2, sixteenth), m8s = __hmul2(s2, __float2half2_rn(-8.0f));
    const uint32_t words[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {        // bytes i, i + 2 of the word: codes 2i, 2i + 4 (low) and 2i + 1, 2i + 5
            const uint32_t x = __byte_perm(words[j], 0x64646464u, i ? 0x4341 : 0x4240), y = x & 0xFFF0FFF0u;
            const __half2 xh = *reinterpret_cast<const __half2 *>(&x), yh = *reinterpret_cast<const __half2 *>(&y);
            const __half2 lo = __hfma2(__hsub2(xh, yh), s2, m8s);
            const __half2 d = __hsub2(yh, k_hi);
            const __half2 hi = SPLIT ? __hmul2(__hmul2(d, sixteenth), s2) : __hmul2(d, s16);
            o[4 * j + 2 * i] = *reinterpret_cast<const uint32_t *>(&lo);
            o[4 * j + 2 * i + 1] = *reinterpret_cast<const uint32_t *>(&hi);
        }
    }
}
// one nibble of each of 16 8-bit codes
__device__ __forceinline__ void eg_convert8(const uint4 &c, uint32_t shift, __half2 s2, uint32_t *o) {
    const __half2 k = __halves2half2(__ushort_as_half(0x6408), __ushort_as_half(0x6408));
    const uint32_t words[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t nib = (words[j] >> shift) & 0x0F0F0F0Fu;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t t = __byte_perm(nib, 0x64646464u, i ? 0x4342 : 0x4140);
            const __half2 q = __hsub2(*reinterpret_cast<const __half2 *>(&t), k);
            const __half2 v = __hmul2(q, s2);
            o[2 * j + i] = *reinterpret_cast<const uint32_t *>(&v);
        }
    }
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t pick_u16(const uint4 &q, uint32_t i) {
    const uint32_t w = (i & 4u) ? ((i & 2u) ? q.w : q.z) : ((i & 2u) ? q.y : q.x);
    return (i & 1u) ? w >> 16 : w & 0xFFFFu;
}

// Correction columns 64 kc .. 64 kc + 63 of one row: [hi | hi | lo | 0], `slots` columns per segment, slot i belonging
// to group i / SPG.  meta: shared-memory address of the row's scales; biases `bias_off` bytes further on.
template <int BITS, int META, int SPG>
__device__ __forceinline__ void eg_correction(uint32_t meta, uint32_t bias_off, uint32_t groups, uint32_t kc, uint32_t (&o)[32]) {
    const float centre = (BITS == 4 ? 8.0f : 136.0f);
    const uint32_t slots = groups * SPG;
    if (slots == (SPG == 1 ? 32u : 16u)) {        // 2048 inputs (phase 0), 512 (phase 1): segments line up with registers
        constexpr int kGroups = SPG == 1 ? 32 : 8;
        const bool want_lo = SPG == 1 && kc == 1u;
#pragma unroll
        for (int v = 0; v < kGroups / 8; ++v) {
            const uint4 sv = lds128(meta + v * 16u), bv = lds128(meta + bias_off + v * 16u);
            const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w}, bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {         // two groups
                const float c0 = fmaf(centre, meta_to_float<META>((uint16_t)sw[i]), meta_to_float<META>((uint16_t)bw[i])) * (1.0f / kBpSumScale);
                const float c1 = fmaf(centre, meta_to_float<META>((uint16_t)(sw[i] >> 16)), meta_to_float<META>((uint16_t)(bw[i] >> 16))) * (1.0f / kBpSumScale);
                const __half2 hi = __floats2half2_rn(c0, c1);
                const float2 hf = __half22float2(hi);
                const __half2 lo = __floats2half2_rn(c0 - hf.x, c1 - hf.y);
                const uint32_t h = *reinterpret_cast<const uint32_t *>(&hi), l = *reinterpret_cast<const uint32_t *>(&lo);
                if (SPG == 1) {
                    o[4 * v + i] = want_lo ? l : h;
                    o[16 + 4 * v + i] = want_lo ? 0u : h;
                } else {                          // both halves of a group have its constant
                    o[2 * i] = __byte_perm(h, h, 0x1010); o[2 * i + 1] = __byte_perm(h, h, 0x3232);
                    o[8 + 2 * i] = o[2 * i]; o[8 + 2 * i + 1] = o[2 * i + 1];
                    o[16 + 2 * i] = __byte_perm(l, l, 0x1010); o[16 + 2 * i + 1] = __byte_perm(l, l, 0x3232);
                    o[24 + 2 * i] = 0u; o[24 + 2 * i + 1] = 0u;
                }
            }
        }
        return;
    }
    const bool vec = (slots & 7u) == 0u && (groups & 7u) == 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {                 // 8 columns at a time
        const uint32_t col0 = kc * 64u + 8u * j;
        float val[8];
        if (vec) {
            const uint32_t seg = col0 / slots, g0 = (col0 - seg * slots) / SPG;     // 8 / SPG groups, one segment
            if (seg < 3u) {
                const uint4 sv = lds128(meta + (g0 & ~7u) * 2u), bv = lds128(meta + bias_off + (g0 & ~7u) * 2u);
#pragma unroll
                for (int e = 0; e < 8 / SPG; ++e) {
                    const uint32_t g = (g0 & 7u) + e;
                    const float cg = fmaf(centre, meta_to_float<META>((uint16_t)pick_u16(sv, g)),
                                          meta_to_float<META>((uint16_t)pick_u16(bv, g))) * (1.0f / kBpSumScale);
                    const float hi = __half2float(__float2half_rn(cg));
                    const float v = seg == 2u ? cg - hi : hi;
#pragma unroll
                    for (int r = 0; r < SPG; ++r) val[e * SPG + r] = v;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) val[e] = 0.0f;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const uint32_t col = col0 + e, seg = col / slots, g = (col - seg * slots) / SPG;
                val[e] = 0.0f;
                if (seg < 3u) {
                    const float cg = fmaf(centre, meta_to_float<META>((uint16_t)lds_u16(meta + 2u * g)),
                                          meta_to_float<META>((uint16_t)lds_u16(meta + bias_off + 2u * g))) * (1.0f / kBpSumScale);
                    const float hi = __half2float(__float2half_rn(cg));
                    val[e] = seg == 2u ? cg - hi : hi;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __half2 h2 = __floats2half2_rn(val[2 * i], val[2 * i + 1]);
            o[4 * j + i] = *reinterpret_cast<const uint32_t *>(&h2);
        }
    }
}

// g / (1 + exp(-g)) through the hardware's approximations (1 to 2 ulp: far below the fp16 operand rounding).  exp overflows to
// infinity and a quotient below 2^-126 is flushed, 0 either way; the intrinsics' handling of subnormal arguments cost a third
// of an epilogue.
__device__ __forceinline__ float eg_silu(float g) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(g * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
    return g * r;
}

// Sum of 8 columns over the 32 lanes: lane l ends up with the sum of column (l >> 2), which column order the halving
// steps below give: bit 4 of the lane picks columns 4-7, bit 3 the upper two of those, bit 2 the upper one.
__device__ __forceinline__ float eg_column_sums(const float (&v)[8], uint32_t lane) {
    float a[4], b[2];
    const bool h16 = (lane & 16u) != 0u, h8 = (lane & 8u) != 0u, h4 = (lane & 4u) != 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = (h16 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, h16 ? v[i] : v[i + 4], 16);
#pragma unroll
    for (int i = 0; i < 2; ++i) b[i] = (h8 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, h8 ? a[i] : a[i + 2], 8);
    float c = (h4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h4 ? b[0] : b[1], 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return c;
}

__device__ __forceinline__ void cp_async16(uint32_t dst_smem, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
// One arrival of this thread on the barrier once its copies so far have landed (the barrier's count includes it).
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// BITS, META: the codes and their scales.  OUT: type of the activations the epilogue of phase 0 makes.
// PHASE 0: gate/up + activation; 1: down.
template <int BITS, int META, int OUT, int PHASE, bool SPLIT>
__global__ void __launch_bounds__(kEgThreads, 1) expert_gemm_kernel(const __grid_constant__ EgArgs args) {
    const EgParams &p = args.p;
    constexpr uint32_t kPasses = (BITS == 8 ? 2u : 1u) * (SPLIT ? 2u : 1u);
    constexpr uint32_t kTiles = PHASE == 0 ? 2u : 1u;             // weight tiles that share a K block of rows
    constexpr uint32_t kStreams = kTiles;                         // threads that issue MMAs, each those of a tile
    constexpr uint32_t kChunkBlocks = BITS == 4 ? 4u : 2u;        // K blocks in a chunk of 128 bytes per row
    constexpr int kSpg = PHASE == 0 ? 1 : 2;                      // correction slots per quantisation group
    extern __shared__ unsigned char eg_smem_raw[];
    const uint32_t raw = smem_addr(eg_smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    EgBarriers *bars = reinterpret_cast<EgBarriers *>(eg_smem_raw + (base - raw));
    const uint32_t chunk_ring = base + 1024u, meta_ring = chunk_ring + kEgChunks * kEgChunkBytes;
    const uint32_t row_ring = base + p.row_ring_off;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const bool all_drain = PHASE == 0 && p.acc_slots == 1u;

    // nothing here (a call whose experts all went to the streaming kernel): out of its way without the set-up
    if (p.list_ready && *p.shared_on == 0u && p.n_work[0] == 0u) {
        pdl_wait();
        pdl_launch_dependents();
        return;
    }

    if (tid == 0) {
        for (uint32_t i = 0; i < 2 * kEgMaxPairs; ++i) { mbar_init(&bars->a_full[i / 2][i % 2], PHASE == 0 ? 4 : 8); mbar_init(&bars->a_empty[i / 2][i % 2], 1); }
        for (uint32_t i = 0; i < kEgChunks; ++i) { mbar_init(&bars->c_full[i], 1); mbar_init(&bars->c_empty[i], kEgProducerWarps); }
        for (uint32_t i = 0; i < kEgMaxMeta; ++i) { mbar_init(&bars->m_full[i], 1); mbar_init(&bars->m_empty[i], kEgProducerWarps); }
        for (uint32_t i = 0; i < kEgMaxRowSlots; ++i) { mbar_init(&bars->b_full[i], PHASE == 0 ? kEgRowWarps * 32 : 1); mbar_init(&bars->b_empty[i], kStreams); }
        for (uint32_t i = 0; i < kEgMaxAcc; ++i) { mbar_init(&bars->d_full[i], kStreams); mbar_init(&bars->d_empty[i], kEgEpilogueWarps + (all_drain ? kEgProducerWarps : 0)); }
        mbar_fence_init();
    }
    if (warp == kEgMmaWarp) {
        tmem_alloc(&bars->tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    constexpr uint32_t tmem = 0;           // an allocation of all 512 columns starts at column 0 (checked below)
    // The rows and what the epilogue reads come from the kernel in front; with list_ready the work list does not, so the
    // code loads and the conversion run ahead of the wait (see stream_gemm_kernel).
    auto wait_in_front = [&]() {
        pdl_wait();
        pdl_launch_dependents();
    };
    if (!p.list_ready) wait_in_front();
    // an earlier wait gave up: do not pile on
    bool ok = __syncthreads_and(*reinterpret_cast<volatile unsigned int *>(p.status) == 0u &&
                                *reinterpret_cast<volatile uint32_t *>(&bars->tmem_slot) == tmem);
    if (p.list_ready && warp >= kEgProducerWarps && warp != kEgCodeWarp) wait_in_front();
    trace_begin(p.trace);

    // bounded by the GPU's nanosecond timer (one second unless a test shortens it), looked at every 16 tries
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (mbar_try_wait_short(bar, parity)) return true;
        const unsigned long long t0 = global_timer_ns(), limit = g_wait_limit_ns;
        for (;;) {
#pragma unroll 1
            for (int it = 0; it < 16; ++it)
                if (mbar_try_wait_short(bar, parity)) return true;
            if (global_timer_ns() - t0 > limit) break;
        }
        atomicExch(p.status, 1u);
        return false;
    };
    // the same for roles with slack (the epilogue, the code loads): they sleep between tries, so that their polling
    // does not take issue slots from the conversion
    auto wait_patient = [&](uint64_t *bar, uint32_t parity) {
        if (mbar_try_wait_short(bar, parity)) return true;
#pragma unroll 1
        for (int it = 0; it < 64; ++it) {
            __nanosleep(100);
            if (mbar_try_wait_short(bar, parity)) return true;
        }
        return wait(bar, parity);
    };

    const uint32_t n_main = p.kdim / 64u;                                     // K blocks of codes
    const uint32_t n_corr = bp_extra_cols(p.kdim, kSpg) / 64u;                // correction K blocks
    const uint32_t n_kb = n_main + n_corr;
    const uint32_t n_mainv = n_main * kPasses, n_v = n_mainv + n_corr;        // A stages per tile
    // One set of accumulators: the MMAs of the next unit wait for them, so the producers, which would wait for those, help the
    // epilogue warps to empty it.
    constexpr uint32_t kDrains = kEgEpilogueWarps / 4, kAllDrains = kDrains + kEgProducerWarps / 4;
    // A slots per sub-unit: phase 0 the two tiles' stages of one K block (and pass), phase 1 two consecutive stages
    const uint32_t n_pair = PHASE == 0 ? n_v : (n_v + 1u) / 2u;
    const uint32_t n_chunk = (n_main + kChunkBlocks - 1u) / kChunkBlocks;     // chunks per tile
    const uint32_t n_sub = PHASE == 0 ? 1u : p.tiles_per_unit;                // accumulator turns per unit
    // the units of the launch: those of the shared items come first, and there are none where another kernel has them
    const uint32_t shared_items = *p.shared_on != 0u ? p.shared_items : 0u;
    const uint32_t total = ok ? (shared_items + p.n_work[0]) * p.units_per_item : 0u;
    const uint32_t meta_bytes = 128u * n_main * 2u;                           // scales (or biases) of a tile

    // v[c] of column c -> half at `at` + c * stride, this lane's place; the lane `partner` away has the half beside it
    auto store_pairs = [&](unsigned char *at, uint32_t stride, uint32_t live, const float (&v)[8], uint32_t partner) {
        const bool upper = (lane & partner) != 0u;
        const uint32_t pick = upper ? 0x3276u : 0x5410u;
        at += upper ? stride - 2u : 0u;
#pragma unroll
        for (uint32_t i = 0; i < 4u; ++i) {
            const __half2 own = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            const uint32_t mine = *reinterpret_cast<const uint32_t *>(&own);
            const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, partner);
            if (2u * i + (upper ? 1u : 0u) < live) *reinterpret_cast<uint32_t *>(at + 2u * i * stride) = __byte_perm(mine, other, pick);
        }
    };
    // Accumulators -> activations / partial rows: every hs-th block of 8 columns from the h-th on, the warp's lane quarter.
    // Two neighbouring columns at a time change hands between the two lanes whose features lie side by side in a row, so
    // that a lane stores two features of one row.
    auto drain = [&](const EgUnit &un, uint32_t sub, uint32_t acc, uint32_t h, uint32_t hs) {
        const uint32_t q = warp & 3u;
        const uint32_t d0 = tmem + ((q * 32u) << 16) + acc * p.acc_stride;
        if (PHASE == 0) {
            const uint32_t f = un.j * 128u + q * 32u + lane;
            // byte offsets inside the unit fit 32 bits
            const uint32_t stride = OUT == OUT_F32 ? p.kfeat * 4u : (p.kfeat + bp_extra_cols(p.kfeat, 2)) * 2u;
            unsigned char *rows = static_cast<unsigned char *>(un.shared ? p.shared_out : p.out) + (size_t)un.start * stride;
            const bool permuted = (un.shared ? p.shared_permute : p.permute) != 0u;
            const uint32_t partner = permuted ? 4u : 1u;       // bp_k_position puts k and k + 4 side by side
            const uint32_t pos = OUT == OUT_F32 ? f * 4u : (permuted ? bp_k_position(f) : f) * 2u;
            const uint32_t slots = p.kfeat / 32u, part = lane & 3u;
            const uint32_t sum_pos = (p.kfeat + part * slots + f / 32u) * 2u;
            for (uint32_t cb = h * 8u; cb < un.count; cb += hs * 8u) {
                uint32_t g8[8], u8[8];
                tmem_ld8(d0 + cb, g8);
                tmem_ld8(d0 + p.acc_tile_off + cb, u8);
                tmem_ld_wait();
                float act[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float g = __uint_as_float(g8[i]), up = __uint_as_float(u8[i]);
                    if (un.shared) { g = round_mid<OUT>(g); up = round_mid<OUT>(up); }     // the shared expert rounds both
                    const float a = p.act == ACT_SILU ? eg_silu(g) : act_gelu_tanh(g);
                    act[i] = round_mid<OUT>(a * up);
                }
                const uint32_t live = min(un.count - cb, 8u);
                if (OUT == OUT_F16) {
                    store_pairs(rows + cb * stride + pos, stride, live, act, partner);
                } else {
                    uint32_t at = cb * stride + pos;
#pragma unroll
                    for (uint32_t i = 0; i < 8u; ++i, at += stride)
                        if (i < live) *reinterpret_cast<float *>(rows + at) = act[i];          // scaled and packed by pack_acts_kernel
                }
                if (OUT == OUT_F16) {          // rows as the down GEMM reads them, with their half-group sums
                    const float sum = eg_column_sums(act, lane) * kBpSumScale;
                    const uint32_t col = lane >> 2;
                    const __half hi = __float2half_rn(sum);
                    const __half lo = __float2half_rn(sum - __half2float(hi));
                    if (part < 3u && col < live)
                        *reinterpret_cast<__half *>(rows + (cb + col) * stride + sum_pos) = part == 1u ? lo : hi;
                }
            }
        } else {
            const uint32_t d = (un.j * n_sub + sub) * 128u + q * 32u + lane;
            const float *scale = un.shared ? p.shared_row_scale : p.row_scale;
            const bool half_out = un.shared ? p.shared_out_half : p.out_half;
            const uint32_t stride = p.out_cols * (half_out ? 2u : 4u), pos = d * (half_out ? 2u : 4u);
            unsigned char *rows = static_cast<unsigned char *>(un.shared ? p.shared_out : p.out) + (size_t)un.start * stride;
            for (uint32_t cb = h * 8u; cb < un.count; cb += hs * 8u) {
                uint32_t r8[8];
                tmem_ld8(d0 + cb, r8);
                tmem_ld_wait();
                const uint32_t live = min(un.count - cb, 8u);
                if (scale != nullptr) {
                    const float mine = scale[un.start + cb + min((uint32_t)lane, live - 1u)];
#pragma unroll
                    for (int i = 0; i < 8; ++i) r8[i] = __float_as_uint(__uint_as_float(r8[i]) * __shfl_sync(0xffffffffu, mine, i));
                }
                if (half_out) {
                    float v[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r8[i]);
                    store_pairs(rows + cb * stride + pos, stride, live, v, 1u);
                } else {
                    uint32_t at = cb * stride + pos;
#pragma unroll
                    for (uint32_t i = 0; i < 8u; ++i, at += stride)
                        if (i < live) *reinterpret_cast<float *>(rows + at) = __uint_as_float(r8[i]);
                }
            }
        }
    };

    if (warp < kEgProducerWarps) {
        // ---------------- producers: codes -> fp16 tiles in tensor memory ----------------
        // group g of four warps: every other A slot from g >> 1 on, stage g & 1 of it (phase 0: the tile; phase 1: the earlier
        // or later stage)
        const uint32_t set = warp >> 3, half = (warp >> 2) & 1u, row = (warp & 3u) * 32u + lane;
        const uint32_t a_dst = (((warp & 3u) * 32u) << 16) + p.a_col + half * kEgStageCols;
        // address of the row's 16-byte piece q in a chunk: (chunk + row_at) ^ (q << 4), the 128-byte swizzle
        const uint32_t row_at = chunk_ring + row * 128u + ((row & 7u) << 4);
        const uint32_t meta_at = meta_ring + row * n_main * 2u;
        const bool vec = (n_main & 7u) == 0u;
        const uint32_t mine_ab = PHASE == 0 ? half : 0u;
        uint32_t pair_base = 0;                    // pairs of the launch so far
        uint32_t slot = set, use = 1;              // A slot of the set's next pair; parity of its refill
        auto next_slot = [&]() { if ((slot += 2u) >= p.a_slots) { slot -= p.a_slots; use ^= 1u; } };
        uint32_t c = 0;                            // chunks of the launch so far (all tiles')
        uint32_t m_slot = 0, m_phase = 0;          // scale tile of the sub-unit (its first one)
        uint32_t d_phase = 0;
        // registers -> the group's stage, once the MMAs that read it last have finished
        auto publish = [&](const uint32_t (&o)[32]) {
            ok = __all_sync(0xffffffffu, wait(&bars->a_empty[slot][mine_ab], use) && ok);
            if (!ok) return;
            tc_fence_after_sync();
            tmem_st32(a_dst + slot * kEgSlotCols, o);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->a_full[slot][mine_ab]);
            next_slot();
        };
        // Of a chunk's K blocks j and passes a group takes every kStep-th block from `first` on, with pass `pass0` (and
        // pass0 + 2 where it has two): its share of the stages in slot order.
        constexpr uint32_t kStep = PHASE == 0 ? (kPasses == 1u ? 2u : 1u) : (kPasses == 1u ? 4u : kPasses == 2u ? 2u : 1u);
        constexpr uint32_t kTwo = PHASE == 0 && kPasses == 4u ? 2u : 1u;
        for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
            for (uint32_t sub = 0; sub < n_sub; ++sub) {
                const uint32_t tile = PHASE == 0 ? half : 0u;
                uint32_t ms = m_slot + tile, mp = m_phase;
                if (ms >= p.meta_slots) { ms -= p.meta_slots; mp ^= 1u; }
                ok = __all_sync(0xffffffffu, wait(&bars->m_full[ms], mp));
                if (!ok) break;
                const uint32_t meta = meta_at + ms * p.meta_slot_bytes;
                const uint32_t par = (pair_base ^ set) & 1u;               // the sub-unit's pairs par, par + 2, ... are this set's
                const uint32_t first = PHASE == 0 ? (kPasses == 1u ? par : 0u) : (kPasses == 1u ? 2u * par + half : kPasses == 2u ? par : 0u);
                const uint32_t pass0 = kPasses == 1u ? 0u : PHASE == 0 ? par : kPasses == 2u ? half : 2u * par + half;
                uint4 scales = make_uint4(0u, 0u, 0u, 0u);
                for (uint32_t m = 0; m < n_chunk; ++m) {
                    const uint32_t mine = (c + tile) % kEgChunks, c_ph = ((c + tile) / kEgChunks) & 1u;
                    uint32_t w[kChunkBlocks / 2];                          // the chunk's scales, two a word
                    if (vec) {
                        constexpr uint32_t kPer = 8u / kChunkBlocks;       // chunks per 8 scales
                        if (m % kPer == 0u) scales = lds128(meta + m / kPer * 16u);
                        if (kChunkBlocks == 4u) {
                            w[0] = (m & 1u) ? scales.z : scales.x; w[kChunkBlocks / 2 - 1] = (m & 1u) ? scales.w : scales.y;
                        } else {
                            w[0] = (m & 2u) ? ((m & 1u) ? scales.w : scales.z) : ((m & 1u) ? scales.y : scales.x);
                        }
                    } else {
#pragma unroll
                        for (uint32_t i = 0; i < kChunkBlocks / 2u; ++i) w[i] = lds32(meta + (m * kChunkBlocks + 2u * i) * 2u);
                    }
                    ok = __all_sync(0xffffffffu, wait(&bars->c_full[mine], c_ph));
                    if (!ok) break;
                    const uint32_t src = (row_at + mine * kEgChunkBytes) ^ (first * (BITS == 4 ? 32u : 64u));
#pragma unroll
                    for (uint32_t i = 0; i < kChunkBlocks / kStep; ++i) {
                        if (m * kChunkBlocks + first + i * kStep >= n_main) break;
                        const uint32_t word = w[(i * kStep) / 2u];
#pragma unroll
                        for (uint32_t t = 0; t < kTwo; ++t) {
                            const uint32_t j = first + i * kStep;
                            const uint32_t wj = kStep == 4u ? ((j & 2u) ? w[kChunkBlocks / 2 - 1] : w[0]) : word;
                            const uint32_t odd = kStep == 1u ? (i & 1u) : (first & 1u);
                            const uint32_t pass = pass0 + 2u * t;
                            const __half2 sc = eg_pass_scale<BITS, META, SPLIT>(wj, odd, pass);
                            uint32_t o[32];
                            if (BITS == 4) {
                                const uint4 a = lds128(src ^ (i * kStep * 32u)), b = lds128(src ^ (i * kStep * 32u + 16u));
                                eg_convert4<SPLIT>(a, b, sc, o);
                            } else {
                                const uint32_t shift = (SPLIT ? pass >> 1 : pass) == 0u ? 4u : 0u;
#pragma unroll
                                for (uint32_t x = 0; x < 4u; ++x) eg_convert8(lds128(src ^ (i * kStep * 64u + (x << 4))), shift, sc, o + 8u * x);
                            }
                            publish(o);
                            if (!ok) break;
                        }
                        if (!ok) break;
                    }
                    if (!ok) break;
                    __syncwarp();                  // (the codes are in registers or further)
                    if ((uint32_t)lane < kTiles) mbar_arrive(&bars->c_empty[(c + lane) % kEgChunks]);
                    c += kTiles;
                }
                if (!ok) break;
                for (uint32_t q = par; q < n_pair; q += 2u) {              // the correction stages among this group's pairs
                    const uint32_t v = PHASE == 0 ? q : 2u * q + half;
                    if (v < n_mainv) { q += (n_mainv - v - 1u) / (PHASE == 0 ? 2u : 4u) * 2u; continue; }
                    if (PHASE == 0 || v < n_v) {
                        uint32_t o[32];
                        eg_correction<BITS, META, kSpg>(meta, meta_bytes, n_main, v - n_mainv, o);
                        publish(o);
                    } else {                       // an odd number of stages: the last slot is half empty
                        ok = __all_sync(0xffffffffu, wait(&bars->a_empty[slot][0], use));
                        if (ok && lane == 0) mbar_arrive(&bars->a_full[slot][0]);
                        next_slot();
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                pair_base += n_pair;
                __syncwarp();
                for (uint32_t t = 0; t < kTiles; ++t) {
                    if (lane == 0) mbar_arrive(&bars->m_empty[m_slot]);
                    if (++m_slot == p.meta_slots) { m_slot = 0; m_phase ^= 1u; }
                }
            }
            if (all_drain && ok) {
                const EgUnit un = eg_unit(p, u, shared_items);
                ok = __all_sync(0xffffffffu, wait(&bars->d_full[0], d_phase));
                d_phase ^= 1u;
                if (!ok) break;
                tc_fence_after_sync();
                drain(un, 0, 0, 2u + (warp >> 2), kAllDrains);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->d_empty[0]);
            }
        }
    } else if (warp == kEgCodeWarp) {
        // ---------------- packed codes and scales: one thread, running ahead ----------------
        if (elect_one()) {
            uint32_t c = 0, m_slot = 0, m_phase = 0;
            for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
                const EgUnit un = eg_unit(p, u, shared_items);
                const uint8_t *blob = p.experts + (size_t)un.expert * p.stride;
                for (uint32_t sub = 0; sub < n_sub && ok; ++sub) {
                    const uint32_t row0 = (PHASE == 0 ? un.j : un.j * n_sub + sub) * 128u;
                    for (uint32_t t = 0; t < kTiles && ok; ++t) {
                        ok = wait_patient(&bars->m_empty[m_slot], m_phase ^ 1u);
                        if (!ok) break;
                        const uint8_t *s = un.shared ? p.shared_s[t] : blob + p.off_s[t];
                        const uint8_t *b = un.shared ? p.shared_b[t] : blob + p.off_b[t];
                        const size_t at = (size_t)row0 * n_main * 2u;
                        unsigned char *dst = eg_smem_raw + (meta_ring - raw) + m_slot * p.meta_slot_bytes;
                        mbar_expect_tx(&bars->m_full[m_slot], 2u * meta_bytes);
                        bulk_g2s(dst, s + at, meta_bytes, &bars->m_full[m_slot]);
                        bulk_g2s(dst + meta_bytes, b + at, meta_bytes, &bars->m_full[m_slot]);
                        if (++m_slot == p.meta_slots) { m_slot = 0; m_phase ^= 1u; }
                    }
                    for (uint32_t k = 0; k < n_chunk && ok; ++k) {
                        for (uint32_t t = 0; t < kTiles && ok; ++t, ++c) {
                            const uint32_t slot = c % kEgChunks;
                            ok = wait_patient(&bars->c_empty[slot], ((c / kEgChunks) & 1u) ^ 1u);
                            if (!ok) break;
                            mbar_expect_tx(&bars->c_full[slot], kEgChunkBytes);
                            const CUtensorMap *map = un.shared ? (t ? &args.shared1 : &args.shared0) : (t ? &args.routed1 : &args.routed0);
                            tma_load_3d(chunk_ring + slot * kEgChunkBytes, map, k * 128u, row0, un.expert, &bars->c_full[slot]);
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp >= kEgRowWarp0 && warp < kEgRowWarp0 + kEgRowWarps) {
        // ---------------- token rows ----------------
        uint32_t slot = 0, phase = 0;
        if (PHASE == 0) {
            // Gathered by 16-byte asynchronous copies (a tensor-map gather of four rows took 80 cycles each, which bound
            // the kernel): lane -> 16-byte piece lane & 7 of rows 16 i + 4 w + (lane >> 3), written where the 128-byte
            // swizzle wants it.  The copies write through the generic proxy; the fence that orders them before the tensor
            // core's reads is the MMA thread's (here it would wait for every copy in flight: 1,000 cycles per K block).
            constexpr int kMaxRows = 12;               // rows per lane: 192 / 16
            const uint32_t w = warp - kEgRowWarp0, piece = lane & 7u, r0 = 4u * w + (lane >> 3);
            const uint32_t dst0 = row_ring + r0 * 128u + ((piece ^ (r0 & 7u)) << 4);
            const uint32_t row_bytes = (p.kdim + bp_extra_cols(p.kdim, 1)) * 2u;
            EgUnit next = eg_unit_or_last(p, blockIdx.x, total, shared_items);
            for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
                const EgUnit un = next;
                const uint32_t n_i = (un.count + 15u) / 16u;
                uint32_t off[kMaxRows];                // byte offsets; rows past the item's end repeat its last one
#pragma unroll
                for (uint32_t i = 0; i < (uint32_t)kMaxRows; ++i) {
                    const uint32_t n = un.start + min(16u * i + r0, un.count - 1u);
                    off[i] = i < n_i ? (un.shared ? n : p.sorted_pair[n] / p.top_k) * row_bytes + piece * 16u : 0u;
                }
                next = eg_unit_or_last(p, u + gridDim.x, total, shared_items);
                const uint8_t *src = reinterpret_cast<const uint8_t *>(un.shared ? p.shared_rows : p.rows);
                for (uint32_t kb = 0; kb < n_kb; ++kb, src += 128) {
                    ok = __all_sync(0xffffffffu, wait(&bars->b_empty[slot], phase ^ 1u));
                    if (!ok) break;
                    if (kb == 2u && !next.shared && (uint32_t)lane * 32u < next.count + 31u)      // its row numbers, into the L1
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(p.sorted_pair + next.start + min(lane * 32u, next.count - 1u)));
                    const uint32_t dst = dst0 + slot * p.row_slot_bytes;
#pragma unroll
                    for (uint32_t b = 0; b < (uint32_t)kMaxRows; b += 3u) {
                        if (b >= n_i) break;
#pragma unroll
                        for (uint32_t i = b; i < b + 3u; ++i)
                            if (i < n_i) cp_async16(dst + i * 2048u, src + off[i]);
                    }
                    const bool drop = p.debug_drop_rows != 0u && kb == 1u && u == 0u;
                    if (!drop) cp_async_arrive(&bars->b_full[slot]);
                    if (++slot == p.row_slots) { slot = 0; phase ^= 1u; }
                }
            }
            cp_async_wait_all();
        } else if (warp == kEgRowWarp0) {
            // consecutive rows: one 16-row box per lane
            for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
                const EgUnit un = eg_unit(p, u, shared_items);
                const uint32_t n_cols = (un.count + 15u) & ~15u;
                const uint32_t loads = p.resident ? 1u : n_sub;
                for (uint32_t sub = 0; sub < loads && ok; ++sub) {
                    for (uint32_t kb = 0; kb < n_kb; ++kb) {
                        ok = __all_sync(0xffffffffu, wait(&bars->b_empty[slot], phase ^ 1u));
                        if (!ok) break;
                        if (lane == 0) mbar_expect_tx(&bars->b_full[slot], n_cols * 128u);
                        __syncwarp();
                        if ((uint32_t)lane * 16u < n_cols)
                            tma_load_2d(row_ring + slot * p.row_slot_bytes + lane * 2048u, un.shared ? &args.shared_rows : &args.rows,
                                        kb * 64u, un.start + lane * 16u, &bars->b_full[slot]);
                        if (++slot == p.row_slots) { slot = 0; phase ^= 1u; }
                    }
                }
            }
        }
    } else if (warp == kEgMmaWarp || warp == kEgMmaWarp1) {
        // ---------------- MMA issue: one thread, phase 0: one per tile ----------------
        if ((PHASE == 0 || warp == kEgMmaWarp) && elect_one()) {
            const uint32_t tile = PHASE == 0 && warp == kEgMmaWarp1 ? 1u : 0u;
            uint32_t st = 0, a_phase = 0;                  // A slot of the next pair
            auto next_pair = [&]() { if (++st == p.a_slots) { st = 0; a_phase ^= 1u; } };
            uint32_t slot = 0, phase = 0, acc = 0, acc_phase = 0;
            const uint64_t db0 = umma_desc_sw128(row_ring);
            const uint32_t slot_step = p.row_slot_bytes >> 4;
            EgUnit next = eg_unit_or_last(p, blockIdx.x, total, shared_items);
            for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
                const EgUnit un = next;
                next = eg_unit_or_last(p, u + gridDim.x, total, shared_items);
                const uint32_t idesc = umma_idesc_f16(128u, (un.count + 15u) & ~15u);
                for (uint32_t sub = 0; sub < n_sub && ok; ++sub) {
                    ok = wait(&bars->d_empty[acc], acc_phase ^ 1u);
                    if (!ok) break;
                    const uint32_t d0 = tmem + acc * p.acc_stride + tile * p.acc_tile_off;
                    if (PHASE == 0) {
                        for (uint32_t kb = 0; kb < n_kb; ++kb) {
                            ok = wait(&bars->b_full[slot], phase);
                            fence_proxy_async_smem();      // rows: generic-proxy writes -> the tensor core's reads
                            const uint64_t db = db0 + (uint64_t)(slot * slot_step);
                            const uint32_t passes = kb < n_main ? kPasses : 1u;
                            for (uint32_t ps = 0; ps < passes; ++ps, next_pair()) {
                                ok = ok && wait(&bars->a_full[st][tile], a_phase);
                                if (!ok) break;
                                tc_fence_after_sync();
                                const uint32_t ta = tmem + p.a_col + st * kEgSlotCols + tile * kEgStageCols;
                                const uint32_t more = (kb | ps) != 0u;
#pragma unroll
                                for (uint32_t k = 0; k < 4u; ++k) {      // 16 values = 8 columns of A = 32 bytes of a row of B
                                    umma_f16_ts(d0, ta + 8u * k, db + 2u * k, idesc, more | k);
                                }
                                umma_commit(&bars->a_empty[st][tile]);
                            }
                            if (!ok) break;
                            umma_commit(&bars->b_empty[slot]);
                            if (++slot == p.row_slots) { slot = 0; phase ^= 1u; }
                        }
                    } else {
                        const bool keep = p.resident && sub + 1u < n_sub;     // the rows serve the next tile too
                        uint32_t bs = slot, bp = phase, kb = 0, ps = 0;
                        for (uint32_t q = 0; q < n_pair; ++q, next_pair()) {
                            ok = wait(&bars->a_full[st][0], a_phase);
                            if (!ok) break;
                            tc_fence_after_sync();
                            const uint32_t ta = tmem + p.a_col + st * kEgSlotCols;
#pragma unroll
                            for (uint32_t t = 0; t < 2u; ++t) {
                                if (2u * q + t >= n_v) break;
                                if (ps == 0u) ok = ok && wait(&bars->b_full[bs], bp);
                                if (!ok) break;
                                const uint64_t db = db0 + (uint64_t)(bs * slot_step);
#pragma unroll
                                for (uint32_t k = 0; k < 4u; ++k)
                                    umma_f16_ts(d0, ta + t * kEgStageCols + 8u * k, db + 2u * k, idesc, 2u * q + t + k);
                                if (++ps == kPasses || kb >= n_main) {
                                    ps = 0; ++kb;
                                    if (!keep) umma_commit(&bars->b_empty[bs]);
                                    if (++bs == p.row_slots) { bs = 0; bp ^= 1u; }
                                }
                            }
                            if (!ok) break;
                            umma_commit(&bars->a_empty[st][0]);
                        }
                        if (!keep) { slot = bs; phase = bp; }
                    }
                    if (!ok) break;
                    umma_commit(&bars->d_full[acc]);
                    if (++acc == p.acc_slots) { acc = 0; acc_phase ^= 1u; }
                }
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const uint32_t h = (warp - kEgProducerWarps) >> 2;
        uint32_t acc = 0, acc_phase = 0;
        EgUnit next = eg_unit_or_last(p, blockIdx.x, total, shared_items);
        for (uint32_t u = blockIdx.x; u < total && ok; u += gridDim.x) {
            const EgUnit un = next;
            next = eg_unit_or_last(p, u + gridDim.x, total, shared_items);
            for (uint32_t sub = 0; sub < n_sub && ok; ++sub) {
                ok = __all_sync(0xffffffffu, wait_patient(&bars->d_full[acc], acc_phase));
                if (!ok) break;
                tc_fence_after_sync();
                drain(un, sub, acc, h, all_drain ? kAllDrains : kDrains);
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->d_empty[acc]);
                if (++acc == p.acc_slots) { acc = 0; acc_phase ^= 1u; }
            }
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    if (!__syncthreads_and(ok)) {          // given up: let the copies and MMAs in flight land before the memory is released
        const unsigned long long t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == kEgMmaWarp) tmem_dealloc(tmem, 512);
    trace_end(p.trace);
}

}  // namespace nvmai
