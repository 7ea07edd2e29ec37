// Kernel launches of the library's translation units.
#pragma once
#include <cuda_runtime.h>
#include <map>
#include <mutex>
#include <utility>

namespace nvmai {

// Kernels here use more than the default 48 KB of dynamic shared memory; the
// opt-in is per function and sticky, so it is raised once per (function, size).
template <typename Kern>
inline cudaError_t ensure_smem(Kern kern, size_t bytes) {
    // the attribute is per device and handles may be driven from several host threads
    static std::map<std::pair<int, const void *>, size_t> granted;
    static std::mutex guard;
    int dev = 0;
    cudaError_t de = cudaGetDevice(&dev);
    if (de != cudaSuccess) return de;
    std::lock_guard<std::mutex> lock(guard);
    const auto key = std::make_pair(dev, reinterpret_cast<const void *>(kern));
    auto it = granted.find(key);
    if (it != granted.end() && it->second >= bytes) return cudaSuccess;
    if (bytes > 40 * 1024) {        // the default limit counts the kernel's static shared memory too
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
    }
    granted[key] = bytes;
    return cudaSuccess;
}

// pdl: launch with programmatic stream serialization, so that the kernel's
// prologue (its weight copies) may overlap the previous kernel's tail.
//
// What every kernel launched here keeps to, and what those that start early lean on:
//   1. Each block waits for the kernel in front (pdl_wait) before it lets the one behind start (pdl_launch_dependents),
//      and no block ends without having waited.  So whatever ran before the kernel in front is complete, and its writes
//      are visible, as soon as a kernel has started at all; the kernel in front itself is complete behind pdl_wait.
//   2. A kernel that puts its own wait off may read, until then, only what kernels before the one in front wrote, and
//      write only what none of them and not the one in front touches: the router GEMM beside the packing of the rows
//      (batch_rows.cuh), a streaming kernel beside the grouped GEMM of the same phase (SgParams::beside).
//      Weights and the work list ahead of the wait (list_ready in batch_path.h) are of this kind.  Tagged words are the exception:
//      stage 3 polls what stage 2 writes (Handover in staged_decode.cuh).
// A kernel that lets its dependents start without having waited would break both without any sign of it.
//
// whole_shared: an SM's split between L1 and shared memory is made for the kernel that runs and cannot change under its blocks, so a
// kernel whose dependents are to fit beside it asks for all of the shared memory.  Asked for launch by launch: as an attribute of the
// function it would also hold for the other handles whose layers the same function runs (six 8-bit layers of one row, 2048 / 768:
// 168 us, behind a handle of 2048 / 128 175).
template <typename Kern, typename... Params>
inline cudaError_t launch_granted(Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl, bool whole_shared,
                                  const Params &...p) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (pdl) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (whole_shared) {
        attr[cfg.numAttrs].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        attr[cfg.numAttrs++].val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    }
    return cudaLaunchKernelEx(&cfg, kern, p...);
}
template <typename Kern, typename... Params>
inline cudaError_t launch_pdl(Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t st, bool pdl, const Params &...p) {
    cudaError_t e = ensure_smem(kern, smem);
    return e != cudaSuccess ? e : launch_granted(kern, grid, block, smem, st, pdl, false, p...);
}

}  // namespace nvmai
