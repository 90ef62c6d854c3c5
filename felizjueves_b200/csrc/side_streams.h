// side_streams.h -- the streams one build spreads its launches over.
#pragma once
#include <cuda_runtime_api.h>

#include <array>
#include <cstddef>
#include <exception>
#include <map>
#include <memory>
#include <mutex>

namespace fjb {

// The side streams a build spreads its class launches over.  A small
// molecule's class kernels each fill a fraction of the GPU for tens of
// microseconds and are independent of one another (they only add into the
// accumulators), so they run side by side: forked off the caller's stream by
// one event, joined back to it by one event a side stream.
struct SideStreams {
    static constexpr int kN = 8;
    cudaStream_t s[kN] = {};
    cudaEvent_t forked = nullptr, joined[kN] = {};
    int priority = 0;   // the streams' priority
    bool lent = false;  // to a call that is enqueuing (StreamPool)
    SideStreams() = default;
    SideStreams(const SideStreams &) = delete;
    SideStreams &operator=(const SideStreams &) = delete;
    cudaError_t make(int prio) {
        priority = prio;
        cudaError_t e = cudaEventCreateWithFlags(&forked, cudaEventDisableTiming);
        for (int i = 0; i < kN && e == cudaSuccess; ++i) {
            e = cudaStreamCreateWithPriority(&s[i], cudaStreamNonBlocking, prio);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&joined[i], cudaEventDisableTiming);
        }
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

// The process's side streams: at most kSets sets a device and stream priority
// (a build's side streams have the priority of the stream it is called on),
// made on first use, however many handles and batches there are, and destroyed
// with the device's last one.  A set is lent to one call for as long as that
// call enqueues; what it has enqueued orders the next borrower behind it
// stream by stream, so callers that build at the same time get sets of their
// own (their slots differ) and only the fifth shares.  A stream that a capture
// has joined belongs to it until the capture ends: such a set is lent to calls
// of the same capture only.
class StreamPool {
public:
    static constexpr int kSets = 4;
    static StreamPool &get() {  // never destroyed: handles may outlive main
        static StreamPool *p = new StreamPool;
        return *p;
    }
    int add_user(int device) {
        std::lock_guard<std::mutex> l(m_);
        ++devices_[device].users;
        return next_slot_++ % kSets;
    }
    void drop_user(int device) {
        std::lock_guard<std::mutex> l(m_);
        auto it = devices_.find(device);
        if (--it->second.users == 0) devices_.erase(it);
    }
    // A set for a call on st, `slot` if that is free; *out null when all are
    // taken.  device is current.
    cudaError_t lend(int device, int slot, cudaStream_t st, SideStreams **out) try {
        *out = nullptr;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        unsigned long long id = 0;
        if (cudaError_t e = cudaStreamGetCaptureInfo(st, &cap, &id)) return e;
        int prio = 0;
        if (cudaError_t e = cudaStreamGetPriority(st, &prio)) return e;
        std::lock_guard<std::mutex> l(m_);
        auto &sets = devices_[device].sets[prio];
        int empty = -1;
        for (int k = 0; k < kSets && !*out && empty != slot; ++k) {
            const int i = (slot + k) % kSets;
            if (!sets[i]) {
                if (empty < 0) empty = i;
                continue;
            }
            if (!sets[i]->lent && usable(*sets[i], cap, id)) *out = sets[i].get();
        }
        if (!*out && empty >= 0) {
            auto fresh = std::make_unique<SideStreams>();
            if (cudaError_t e = make_uncaptured(*fresh, prio)) return e;
            sets[empty] = std::move(fresh);
            *out = sets[empty].get();
        }
        if (*out) (*out)->lent = true;
        return cudaSuccess;
    } catch (const std::exception &) {  // out of host memory, at a C entry
        return cudaErrorMemoryAllocation;
    }
    void give_back(SideStreams *s) {
        std::lock_guard<std::mutex> l(m_);
        s->lent = false;
    }

private:
    struct Device {
        int users = 0;
        std::map<int, std::array<std::unique_ptr<SideStreams>, kSets>> sets;  // by priority
    };
    std::mutex m_;
    std::map<int, Device> devices_;
    unsigned next_slot_ = 0;

    // Making streams and events is not work that a running capture records:
    // a call captured before any eager one gets its set too.
    static cudaError_t make_uncaptured(SideStreams &s, int prio) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        if (cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode)) return e;
        const cudaError_t e = s.make(prio), back = cudaThreadExchangeStreamCaptureMode(&mode);
        return e != cudaSuccess ? e : back;
    }
    // not part of a capture, or of the caller's own
    static bool usable(const SideStreams &s, cudaStreamCaptureStatus cap, unsigned long long id) {
        cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
        unsigned long long sid = 0;
        if (cudaStreamGetCaptureInfo(s.s[0], &c, &sid) != cudaSuccess) return false;
        if (c == cudaStreamCaptureStatusNone) return true;
        return c == cudaStreamCaptureStatusActive && cap == cudaStreamCaptureStatusActive && sid == id;
    }
};

// A handle's or batch's place in the pool.
class StreamUser {
    int device_ = -1, slot_ = 0;

public:
    StreamUser() = default;
    StreamUser(const StreamUser &) = delete;
    StreamUser &operator=(const StreamUser &) = delete;
    ~StreamUser() {
        if (device_ >= 0) StreamPool::get().drop_user(device_);
    }
    void attach(int device) {
        slot_ = StreamPool::get().add_user(device);
        device_ = device;
    }
    cudaError_t lend(cudaStream_t st, SideStreams **out) {
        return StreamPool::get().lend(device_, slot_, st, out);
    }
};

// One fork off a caller's stream: joined back to it by join(), and by the end
// of the scope on every other way out -- a return between fork and join would
// leave kernels on streams that the caller's stream, and so its allocator,
// does not wait for.  user null, or no set free: every at() is the caller's
// stream.
class Fork {
    StreamUser *user_;
    SideStreams *side_ = nullptr;
    cudaStream_t st_;

public:
    Fork(StreamUser *user, cudaStream_t st) : user_(user), st_(st) {}
    Fork(const Fork &) = delete;
    Fork &operator=(const Fork &) = delete;
    ~Fork() { join(); }
    cudaError_t begin() {
        if (!user_) return cudaSuccess;
        if (cudaError_t e = user_->lend(st_, &side_)) return e;
        return side_ ? side_->fork(st_) : cudaSuccess;
    }
    cudaError_t join() {
        if (!side_) return cudaSuccess;
        const cudaError_t e = side_->join(st_);
        StreamPool::get().give_back(side_);
        side_ = nullptr;
        return e;
    }
    cudaStream_t at(size_t i) const { return side_ ? side_->s[i % SideStreams::kN] : st_; }
};

}  // namespace fjb
