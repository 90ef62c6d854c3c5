// side_streams.h -- the streams one build spreads its launches over.
#pragma once
#include <cuda_runtime.h>

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
    cudaError_t join(cudaStream_t st) {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < kN && e == cudaSuccess; ++i) {
            e = cudaEventRecord(joined[i], s[i]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(st, joined[i], 0);
        }
        return e;
    }
    ~SideStreams() {
        for (int i = 0; i < kN; ++i) {
            if (s[i]) cudaStreamDestroy(s[i]);
            if (joined[i]) cudaEventDestroy(joined[i]);
        }
        if (forked) cudaEventDestroy(forked);
    }
};

}  // namespace fjb
