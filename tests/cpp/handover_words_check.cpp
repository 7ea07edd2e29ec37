// The hand-over's tags against a CUDA runtime that works on host memory: a call never meets a word of an earlier call with its own
// tag, however many calls there have been, and a handle without memory for the words goes without.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

static bool no_memory, no_clear;
static int cleared;

extern "C" cudaError_t cudaMalloc(void **p, size_t bytes) {
    *p = no_memory ? nullptr : std::malloc(bytes);
    if (*p != nullptr) std::memset(*p, 0x5A, bytes);
    return *p != nullptr ? cudaSuccess : cudaErrorMemoryAllocation;
}
extern "C" cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
extern "C" cudaError_t cudaMemsetAsync(void *p, int v, size_t bytes, cudaStream_t) {
    if (no_clear) return cudaErrorUnknown;
    ++cleared;
    std::memset(p, v, bytes);
    return cudaSuccess;
}
extern "C" cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *) { return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

#include "../../nvmai_b200/csrc/handover_words.h"

int main() {
    int bad = 0;
    auto expect = [&](const char *what, bool ok) { if (!ok) { std::printf("%s\n", what); ++bad; } };
    nvmai::HandoverWords none, h;
    expect("no words, no tag", h.next_tag(nullptr) == 0);
    no_memory = true;
    none.make(96, nullptr);
    no_memory = false;
    none.make(96, nullptr);
    expect("asked for memory once, without success", none.words() == nullptr && none.next_tag(nullptr) == 0);
    h.make(96, nullptr);
    unsigned long long *words = h.words();
    h.make(96, nullptr);
    expect("memory, cleared, once", words != nullptr && h.words() == words && words[0] == 0 && words[95] == 0);
    cleared = 0;
    // a call of n rows of 32 words: none has the call's tag before it is written, then all of the call's do
    auto call = [&](int n) {
        const uint32_t tag = h.next_tag(nullptr);
        expect("a tag", tag != 0);
        for (int i = 0; i < 96; ++i) expect("a word of an earlier call has the tag", (uint32_t)(h.words()[i] >> 32) != tag);
        for (int i = 0; i < 32 * n; ++i) h.words()[i] = (unsigned long long)tag << 32;
    };
    for (int i = 0; i < 5; ++i) call(3);           // three rows leave the tags 1 to 5 in the words of rows 1 and 2
    expect("nothing cleared yet", cleared == 0);
    h.skip_to(nvmai::HandoverWords::kLastTag - 2);
    for (int i = 0; i < 6; ++i) call(1);           // one row only, past the last tag and up to 4
    for (int i = 0; i < 8; ++i) call(3);
    expect("cleared once", cleared == 1);
    h.skip_to(nvmai::HandoverWords::kLastTag);
    no_clear = true;
    expect("words that could not be cleared are not used", h.next_tag(nullptr) == 0 && h.next_tag(nullptr) == 0);
    no_clear = false;
    call(2);
    h.release();
    expect("released", h.words() == nullptr && h.next_tag(nullptr) == 0);
    std::printf(bad ? "FAILED %d\n" : "PASSED\n", bad);
    return bad != 0;
}
