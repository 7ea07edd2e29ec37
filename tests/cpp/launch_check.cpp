// Launches through launch.h against a CUDA runtime that only takes notes: which attributes a launch has, and which of them
// stick to the function.
#include <cuda_runtime.h>

#include <cstdio>

static int function_attributes, largest_smem;
static bool launch_pdl_on, launch_whole;

extern "C" cudaError_t cudaGetDevice(int *dev) { *dev = 0; return cudaSuccess; }
// (the headers have this template for nvcc only)
template <typename T>
cudaError_t cudaFuncSetAttribute(T *, cudaFuncAttribute attr, int value) {
    if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) largest_smem = value;
    else ++function_attributes;
    return cudaSuccess;
}
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *cfg, const void *, void **) {
    launch_pdl_on = launch_whole = false;
    for (unsigned i = 0; i < cfg->numAttrs; ++i) {
        const cudaLaunchAttribute &a = cfg->attrs[i];
        if (a.id == cudaLaunchAttributeProgrammaticStreamSerialization) launch_pdl_on = a.val.programmaticStreamSerializationAllowed == 1;
        if (a.id == cudaLaunchAttributePreferredSharedMemoryCarveout) launch_whole = a.val.sharedMemCarveout == (unsigned)cudaSharedmemCarveoutMaxShared;
    }
    return cudaSuccess;
}

#include "../../nvmai_b200/csrc/launch.h"

static void kernel(int) {}

int main() {
    int bad = 0;
    // two handles' launches of one function, in either order: each has its own split, whatever ran before it
    const struct { size_t smem; bool pdl, whole; } launches[] = {
        {100 << 10, true, false}, {60 << 10, true, true}, {60 << 10, false, true}, {100 << 10, true, false}, {200 << 10, false, false}, {60 << 10, true, true}};
    int most = 0;
    for (const auto &l : launches) {
        cudaError_t e = nvmai::ensure_smem(kernel, l.smem);
        if (e == cudaSuccess) e = nvmai::launch_granted(kernel, dim3(1), dim3(32), l.smem, nullptr, l.pdl, l.whole, 1);
        most = l.smem > (size_t)most ? (int)l.smem : most;
        bad += e != cudaSuccess || launch_pdl_on != l.pdl || launch_whole != l.whole || function_attributes != 0 || largest_smem != most;
    }
    std::printf(bad ? "FAILED %d\n" : "PASSED\n", bad);
    return bad != 0;
}
