// side_streams.h -- the streams one build spreads its launches over.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>

namespace fjb {

// The side streams a build spreads its class launches over.  A small
// molecule's class kernels each fill a fraction of the GPU for tens of
// microseconds and are independent of one another (they only add into the
// accumulators), so they run side by side: forked off the caller's stream by
// one event, joined back to it by one event a side stream.  Owned by one
// handle or batch, like its accumulators.
struct SideStreams {
    static constexpr int kN = 8;
    cudaStream_t s[kN] = {};
    cudaEvent_t forked = nullptr, joined[kN] = {};
    bool ready = false;
    cudaError_t ensure() {
        if (ready) return cudaSuccess;
        cudaError_t e = forked ? cudaSuccess : cudaEventCreateWithFlags(&forked, cudaEventDisableTiming);
        for (int i = 0; i < kN && e == cudaSuccess; ++i) {
            if (!s[i]) e = cudaStreamCreateWithFlags(&s[i], cudaStreamNonBlocking);
            if (e == cudaSuccess && !joined[i]) e = cudaEventCreateWithFlags(&joined[i], cudaEventDisableTiming);
        }
        ready = e == cudaSuccess;
        return e;
    }
    cudaError_t fork(cudaStream_t st) {
        cudaError_t e = cudaEventRecord(forked, st);
        for (int i = 0; i < kN && e == cudaSuccess; ++i) e = cudaStreamWaitEvent(s[i], forked, 0);
        return e;
    }
    // st waits for every side stream, whatever fails on the way.
    cudaError_t join(cudaStream_t st) {
        cudaError_t first = cudaSuccess;
        for (int i = 0; i < kN; ++i) {
            cudaError_t e = cudaEventRecord(joined[i], s[i]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(st, joined[i], 0);
            if (first == cudaSuccess) first = e;
        }
        return first;
    }
    ~SideStreams() {
        for (int i = 0; i < kN; ++i) {
            if (s[i]) cudaStreamDestroy(s[i]);
            if (joined[i]) cudaEventDestroy(joined[i]);
        }
        if (forked) cudaEventDestroy(forked);
    }
};

// One fork off a caller's stream: joined back to it by join(), and by the end
// of the scope on every other way out -- a return between fork and join would
// leave kernels on streams that the caller's stream, and so its allocator,
// does not wait for.  side null: every at() is the caller's stream.
class Fork {
    SideStreams *side_;
    cudaStream_t st_;
    bool open_ = false;

public:
    Fork(SideStreams *side, cudaStream_t st) : side_(side), st_(st) {}
    Fork(const Fork &) = delete;
    Fork &operator=(const Fork &) = delete;
    ~Fork() { join(); }
    cudaError_t begin() {
        open_ = side_ != nullptr;
        return open_ ? side_->fork(st_) : cudaSuccess;
    }
    cudaError_t join() {
        if (!open_) return cudaSuccess;
        open_ = false;
        return side_->join(st_);
    }
    cudaStream_t at(size_t i) const { return side_ ? side_->s[i % SideStreams::kN] : st_; }
};

}  // namespace fjb
