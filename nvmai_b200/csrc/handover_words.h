// Device memory of the decode stages' hand-over (Handover in staged_decode.cuh) and the tags of its calls.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace nvmai {

class HandoverWords {
public:
    // With the first call that uses them, once, also where there is no memory for them; another stream's capture is not disturbed.
    // (10 us of that call.  Made with the handle or its first layer, by handles that never use them too, they move what is allocated
    // next: a 40-layer step of the resident kernel 607 -> 625 us; in 2 MB of their own it stays, for 0.4 ms of set-up.)
    void make(size_t count, cudaStream_t st) {
        if (asked_) return;
        asked_ = true;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (cudaMalloc(reinterpret_cast<void **>(&words_), count * sizeof(*words_)) == cudaSuccess &&
            cudaMemsetAsync(words_, 0, count * sizeof(*words_), st) == cudaSuccess) {
            count_ = count;
        } else {
            cudaGetLastError();
            release();
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    void release() {
        cudaFree(words_);
        words_ = nullptr;
        count_ = 0;
    }
    unsigned long long *words() const { return words_; }
    // A tag that no word has: 1, 2, ...  Once all have been given out the words are cleared, behind the calls before this one.  0: none.
    uint32_t next_tag(cudaStream_t st) {
        if (words_ == nullptr) return 0;
        if (tag_ == kLastTag) {
            if (cudaMemsetAsync(words_, 0, count_ * sizeof(*words_), st) != cudaSuccess) {
                cudaGetLastError();
                return 0;
            }
            tag_ = 0;
        }
        return ++tag_;
    }
    void skip_to(uint32_t tag) { tag_ = tag; }      // (for tests)

    static constexpr uint32_t kLastTag = 0xFFFFFFFFu;

private:
    unsigned long long *words_ = nullptr;
    size_t count_ = 0;
    uint32_t tag_ = 0;
    bool asked_ = false;
};

}  // namespace nvmai
