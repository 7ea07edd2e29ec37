// Interface between the C ABI's translation unit and the batched path's (prefill chunks and larger decode batches):
// the kernels' parameter blocks and their launchers.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace nvmai {

struct WorkItem { uint32_t expert, start, count, pad; };

// Extra K columns that carry the affine correction: 3 fp16 values per slot (`spg` slots per quantisation group of 64
// values), rounded up to K blocks of 64.
__host__ __device__ constexpr uint32_t bp_extra_cols(uint32_t kdim, uint32_t spg) {
    return ((3u * spg * (kdim / 64u) + 63u) / 64u) * 64u;
}
// The group sums in the correction columns are stored times this factor (and the constants they multiply divided by
// it): 64 fp16 values can add up to 2^22.
constexpr float kBpSumScale = 1.0f / 128.0f;
// Order in which the 4-bit unpack delivers the 8 codes of a word (position -> K index), and where a K index lands.
__host__ __device__ constexpr uint32_t bp_k_order(uint32_t pos) { return ((pos & 1u) << 2) | (pos >> 1); }
__host__ __device__ constexpr uint32_t bp_k_position(uint32_t k) { return (k & ~7u) | ((k & 3u) << 1) | ((k & 7u) >> 2); }

// ---- grouped expert GEMMs (expert_gemm.cuh) ------------------------------------------------
struct EgParams {
    const uint8_t *experts; unsigned long long stride; uint32_t num_experts;
    uint32_t off_s[2], off_b[2];              // scales, biases inside a blob: phase 0 gate, up; phase 1 down
    const uint8_t *shared_s[2], *shared_b[2];
    const WorkItem *work; const uint32_t *n_work; const uint32_t *sorted_pair;
    const __half *rows, *shared_rows;         // phase 0: x rows with their correction columns (phase 1: the tensor maps)
    uint32_t shared_items;                    // items 0 .. shared_items - 1 are even runs of token rows (shared expert)
    const uint32_t *shared_on;                // none of them if this word is 0
    uint32_t units_per_item, tiles_per_unit;  // phase 0: F / 128, -; phase 1: D / 128 / tiles_per_unit, tiles_per_unit
    uint32_t tokens, top_k, cap;              // cap: most rows of an item
    uint32_t kdim;                            // D (phase 0) / F (phase 1)
    uint32_t kfeat, out_cols;                 // phase 0: F; phase 1: D
    void *out, *shared_out;                   // phase 0: activations; phase 1: partial rows
    uint32_t out_half, shared_out_half;       // phase 1: fp16 partial rows instead of fp32
    uint32_t permute, shared_permute;         // phase 0, fp16 activations: the down weights' K order is the 4-bit unpack's
    const float *row_scale, *shared_row_scale;    // phase 1: factor per row undone in the epilogue, or nullptr
    uint32_t act;
    uint32_t resident;                        // phase 1: an item's rows fit the ring and stay for all tiles of a unit
    uint32_t row_slots, row_slot_bytes, row_ring_off, meta_slots, meta_slot_bytes;
    uint32_t acc_slots, acc_stride, acc_tile_off;
    uint32_t a_slots, a_col;                  // A slots and the tensor-memory column of the first one (the last ends at 512)
    uint32_t list_ready;                      // 1: the work list was complete before the kernel in front of this one could start
    uint32_t debug_drop_rows;                 // test hook: block 0 never announces its second K block of rows, so waits run out
    unsigned int *status;
    unsigned long long *trace;
};
struct alignas(64) EgArgs {
    CUtensorMap routed0, routed1;             // codes [experts][rows][bytes]: gate, up / down
    CUtensorMap shared0, shared1;
    CUtensorMap rows, shared_rows;            // phase 1: activation rows with their correction columns
    EgParams p;
};
constexpr uint32_t kEgChunks = 4;             // ring of 16 KB pieces of packed codes
struct EgPlan { uint32_t cap; size_t smem; };
// Fills the ring geometry of p for rows of p.kdim values and items of up to want_cap rows; cap = 0: does not fit.
EgPlan eg_plan(EgParams &p, int phase, uint32_t want_cap);
cudaError_t eg_launch(int phase, uint32_t bits, uint32_t meta, uint32_t out_dtype, bool split, const EgArgs &args, uint32_t blocks,
                      size_t smem, cudaStream_t st);

// ---- few rows per expert: codes streamed through mma.sync (stream_gemm.cuh) -----------------
struct SgParams {
    const uint8_t *experts; unsigned long long stride; uint32_t num_experts;
    uint32_t off_s[2], off_b[2];
    const uint8_t *shared_s[2], *shared_b[2];
    const void *rows, *shared_rows;           // phase 0: fp16 x rows [token][kdim]; phase 1: activation rows (fp16 / fp32)
    const WorkItem *work; const uint32_t *n_work; const uint32_t *sorted_pair;
    const uint32_t *shared_on;                // 0 there: no shared items
    uint32_t shared_items, units_per_item, tokens, top_k, cap, kdim, out_cols, act;
    void *out, *shared_out;                   // phase 0: activations [row][F]; phase 1: fp32 partial rows [row][D]
    uint32_t stages, meta_off, meta_bytes, x_off, raw_off, sum_off, scale_off;
    uint32_t list_ready;                      // as in EgParams
    uint32_t beside;                          // 1: runs beside the kernel in front of it, needs only what that one waited for
    unsigned int *status;
};
struct alignas(64) SgArgs {
    CUtensorMap routed0, routed1, shared0, shared1;     // codes, boxes of 64 rows x 128 bytes
    SgParams p;
};
// Fills the shared-memory geometry of p (kdim and out_cols set) for items of up to 8 * nb rows; 0: does not fit.
size_t sg_plan(SgParams &p, int phase, uint32_t nb, bool wide);
cudaError_t sg_launch(int phase, uint32_t bits, uint32_t meta, uint32_t out_dtype, uint32_t nb, const SgArgs &args, uint32_t blocks,
                      size_t smem, cudaStream_t st);

// ---- rows, routing and reduction around them (batch_rows.cuh) --------------------------------
// x rows -> fp16 rows in the weights' K order with their group sums; optionally the scalar gate of every row
struct PackXParams {
    const __half *x; __half *dst, *dst2;      // dst2: a second copy in the other K order (nullptr: none)
    uint32_t rows, n, permute;                // dst's K order: 1 = the 4-bit unpack's; dst2 has the other one
    const __half *gate_row; float *gate_val;  // dense fp16 gate row [n], nullptr: none
    uint32_t out_half;                        // rounding of gate_val: 1 = half, 0 = 11 significant bits
};
cudaError_t bp_pack_x(const PackXParams &p, cudaStream_t st);

// dense fp16 router: logits as partial sums [term][tokens][experts]
struct RouterParams { float *logits; uint32_t tokens, experts, kdim, splits; unsigned int *status; };
struct alignas(64) RouterArgs { CUtensorMap w, x; RouterParams p; };
constexpr uint32_t kRouterTileTokens = 64;
constexpr uint32_t kRouterParts = 4;      // quarters of K that the logits add up from; splits: 1, 2 or 4 blocks share them
inline uint32_t bp_router_terms(uint32_t splits) { return splits == 1 ? 1 : splits == 2 ? 3 : 4; }     // see router_gemm_kernel
cudaError_t bp_router(const RouterArgs &args, cudaStream_t st);

// top-k of every row (or the given experts), histograms per block, and in the last block the scan: offsets per expert,
// first positions per block, the GEMMs' work lists
struct RouteParams {
    const float *logits; uint32_t terms;      // [term][tokens][E], 1 to 4 terms; nullptr: idx is given
    const uint16_t *pes;
    uint32_t *idx; __half *w;
    uint32_t tokens, E, K;
    const uint32_t *expert_map; uint32_t n_local;
    uint16_t *block_hist;                     // [block][kMaxExperts] pairs
    // [segment of blocks][kMaxExperts]: an expert's pairs (zero between calls); its first row and, behind the first segment's, the
    // pairs of the segments in front
    uint32_t *totals, *first;
    unsigned int *counter;
    uint32_t *sorted_pair, *inv;
    // work lists: 0, 1 the grouped GEMMs' (gate/up, down) of the experts with more than `heavy` rows, 2 the streaming
    // kernel's of the others (both phases).  `heavy` is taken as "none" where those experts hold fewer than
    // `heavy_min` pairs; shared_on[0] / [1]: 1 if the grouped GEMMs / the streaming kernel have the shared expert.
    uint32_t *shared_on;
    WorkItem *work[3]; uint32_t *n_work[3]; uint32_t cap[3]; uint32_t heavy, heavy_min;
};
uint32_t bp_route_blocks(uint32_t tokens);
constexpr uint32_t kRouteSegment = 128;       // routing blocks whose counts a block of the scatter adds up itself
__host__ __device__ constexpr uint32_t bp_route_segments(uint32_t blocks) { return (blocks + kRouteSegment - 1u) / kRouteSegment; }
constexpr uint32_t kSmallRoute = 32;          // up to this many tokens one block does it all
cudaError_t bp_route(const RouteParams &p, cudaStream_t st);
inline uint64_t bp_route_launches(uint32_t tokens) { return tokens <= kSmallRoute ? 1 : 2; }

// wide-range activations: fp32 rows -> scaled fp16 rows in the down weights' K order with half-group sums
// (routed rows, then the shared expert's)
struct PackActsParams {
    const float *src; __half *dst; float *row_scale; uint32_t rows, n, permute;
    const float *src2; __half *dst2; float *row_scale2; uint32_t rows2, n2, permute2;
};
cudaError_t bp_pack_acts(const PackActsParams &p, cudaStream_t st);

constexpr uint32_t kBpNormRow = 2048;     // longest row that the reduction normalises itself
struct CombineRowsParams {
    const void *partial; uint32_t partial_half;
    const void *shared_partial; uint32_t shared_half;     // nullptr: no shared expert
    const uint32_t *inv; const __half *routing_w; const float *gate_val;
    void *y, *hidden;
    const __half *hidden_delta;   // decode order only
    float *partial_y;             // this rank's share only
    __half *x_next;               // or nullptr: the next block's input, half(y * rsqrt(mean(y^2) + 1e-6)); D <= kBpNormRow, decode order
    uint32_t tokens, D, K, prefill;
    uint32_t sms;                 // SMs of the device
    uint32_t aligned;             // set by bp_combine
};
cudaError_t bp_combine(const CombineRowsParams &p, uint32_t out_dtype, cudaStream_t st);

cudaError_t bp_set_wait_limit(unsigned long long ns);

}  // namespace nvmai
