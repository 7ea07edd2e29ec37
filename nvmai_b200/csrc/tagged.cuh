// Values that cross blocks without a kernel boundary or a barrier: 64-bit words {payload, tag}, written in one store and
// polled until the tag matches, so that the data arrives with its flag (see persistent_decode.cuh, staged_decode.cuh).
#pragma once
#include "tma.cuh"

namespace nvmai {

__device__ __forceinline__ void st_tagged(unsigned long long *p, uint32_t tag, float v) {
    const unsigned long long w = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void st_tagged_bits(unsigned long long *p, uint32_t tag, uint32_t v) { st_tagged(p, tag, __uint_as_float(v)); }
__device__ __forceinline__ unsigned long long ld_tagged(const unsigned long long *p) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ void ld_tagged2(const unsigned long long *p, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool tag_is(unsigned long long w, uint32_t tag) { return (uint32_t)(w >> 32) == tag; }
__device__ __forceinline__ float tag_val(unsigned long long w) { return __uint_as_float((uint32_t)w); }

// Time limit of a polling loop: looks at the clock and at the status word (another
// block has already given up) once in a while.
struct PollClock {
    unsigned long long t0 = 0;
    uint32_t spins = 0;
    __device__ __forceinline__ bool expired(const unsigned int *status) {
        if ((++spins & 31u) != 0) return false;
        if (*reinterpret_cast<const volatile unsigned int *>(status) != 0) return true;
        const unsigned long long now = global_timer_ns();
        if (t0 == 0) { t0 = now; return false; }
        return now - t0 > g_wait_limit_ns;
    }
};

__device__ __forceinline__ bool poll_tagged(const unsigned long long *p, uint32_t tag, float &v, unsigned int *status) {
    PollClock clk;
    for (;;) {
        const unsigned long long w = ld_tagged(p);
        if (tag_is(w, tag)) { v = tag_val(w); return true; }
        if (clk.expired(status)) { atomicExch(status, 1u); return false; }
    }
}

// out[j] = the value of word first + j * STRIDE of src (j < N, index below limit; 0 for the others), each waited for
// until it carries `tag`.  A round requests every word still missing before it looks at any, so the requests overlap
// (one L2 round trip per round instead of one per word).
template <int N, int STRIDE>
__device__ __forceinline__ bool poll_strided(const unsigned long long *src, int first, int limit, uint32_t tag, float (&out)[N],
                                             unsigned int *status) {
    static_assert(N <= 32, "one pending bit per word");
    uint32_t pending = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        out[j] = 0.0f;
        if (first + j * STRIDE < limit) pending |= 1u << j;
    }
    PollClock clk;
    while (pending) {
        const uint32_t round = pending;
        unsigned long long w[N];
#pragma unroll
        for (int j = 0; j < N; ++j) w[j] = (round >> j) & 1u ? ld_tagged(src + first + j * STRIDE) : 0ull;
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (((round >> j) & 1u) && tag_is(w[j], tag)) { out[j] = tag_val(w[j]); pending &= ~(1u << j); }
        if (pending && clk.expired(status)) { atomicExch(status, 1u); return false; }
    }
    return true;
}

}  // namespace nvmai
