// The stream fork (side_streams.h) on the CPU: the CUDA calls it makes are
// counted by the stand-ins below instead of the runtime.  Prints "ok" or the
// first thing that is wrong; built and run by tests/test_side_streams.py.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "side_streams.h"

using namespace fjb;

// what the stand-in runtime saw
static std::recursive_mutex g_m;
static int g_streams, g_events, g_launches;          // live streams and events, launches so far
static std::map<cudaStream_t, int> g_last;           // a stream's last launch
static std::map<cudaEvent_t, std::map<cudaStream_t, int>> g_event;  // what an event covers
static std::map<cudaStream_t, std::map<cudaStream_t, int>> g_seen;  // what a stream has waited for
static std::map<cudaStream_t, int> g_prio;           // a stream's priority
static std::map<cudaStream_t, unsigned long long> g_cap;  // the capture a stream is part of
static std::map<cudaEvent_t, unsigned long long> g_ecap;  // and an event was recorded in
static thread_local bool g_relaxed;  // the thread's capture mode
static int g_fail_at = -1, g_calls;                       // the call that fails, if any

static cudaError_t call() { return g_calls++ == g_fail_at ? cudaErrorUnknown : cudaSuccess; }
static void need(bool ok, const char *what) {
    if (ok) return;
    std::printf("%s\n", what);
    std::exit(1);
}
#define LOCKED std::lock_guard<std::recursive_mutex> lock(g_m)

extern "C" {
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int prio) {
    LOCKED;
    need(g_relaxed, "a stream made in a mode in which a capture refuses it");
    *s = (cudaStream_t)std::malloc(1);
    g_prio[*s] = prio;
    ++g_streams;
    return cudaSuccess;
}
cudaError_t cudaStreamGetPriority(cudaStream_t s, int *prio) {
    LOCKED;
    *prio = g_prio[s];
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    LOCKED;
    g_cap.erase(s);
    g_prio.erase(s);
    g_last.erase(s);
    g_seen.erase(s);
    std::free(s);
    --g_streams;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    LOCKED;
    *e = (cudaEvent_t)std::malloc(1);
    ++g_events;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    LOCKED;
    g_event.erase(e);
    g_ecap.erase(e);
    std::free(e);
    --g_events;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    LOCKED;
    if (cudaError_t r = call()) return r;
    g_event[e] = g_seen[s];
    g_event[e][s] = g_last[s];
    g_ecap[e] = g_cap[s];
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    LOCKED;
    if (cudaError_t r = call()) return r;
    for (auto &kv : g_event[e])
        if (kv.second > g_seen[s][kv.first]) g_seen[s][kv.first] = kv.second;
    need(!g_cap[s] || g_cap[s] == g_ecap[e], "a call outside a capture, or of another, took one of its streams");
    if (g_ecap[e]) g_cap[s] = g_ecap[e];
    return cudaSuccess;
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus *st, unsigned long long *id,
                                     cudaGraph_t *, const cudaGraphNode_t **, size_t *) {
    LOCKED;
    *id = g_cap[s];
    *st = *id ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
}
extern "C" cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode *m) {
    LOCKED;
    const bool was = g_relaxed;
    g_relaxed = *m == cudaStreamCaptureModeRelaxed;
    *m = was ? cudaStreamCaptureModeRelaxed : cudaStreamCaptureModeThreadLocal;
    return cudaSuccess;
}
static void end_capture(unsigned long long id) {
    for (auto &kv : g_cap)
        if (kv.second == id) kv.second = 0;
}

static void launch(cudaStream_t s) { g_last[s] = ++g_launches; }
// st waits for every launch so far
static bool joined(cudaStream_t st, const std::set<cudaStream_t> &used) {
    for (cudaStream_t s : used)
        if (s != st && g_seen[st][s] < g_last[s]) return false;
    return true;
}

static cudaStream_t const kCaller = (cudaStream_t)0x10;

// a call that forks, launches n kernels and returns (early: without join)
static int build(StreamUser *user, int n, bool early, std::set<cudaStream_t> *used) {
    Fork fork(user, kCaller);
    if (fork.begin() != cudaSuccess) return 1;
    for (int i = 0; i < n; ++i) {
        used->insert(fork.at(i));
        launch(fork.at(i));
    }
    if (early) return 1;
    return fork.join() != cudaSuccess;
}

static void test_joins() {
    StreamUser side;
    side.attach(0);
    for (int n : {0, 1, 5, 20})
        for (bool early : {false, true}) {
            std::set<cudaStream_t> used;
            launch(kCaller);
            need(build(&side, n, early, &used) == early, "status");
            need(joined(kCaller, used), "a way out left a side stream unjoined");
            for (cudaStream_t s : used) need(g_seen[s][kCaller] == g_last[kCaller], "a side stream did not wait");
        }
    // a failing call in the fork or the join: the streams it does not touch are joined
    for (int at = 0; at < 2 * (1 + 2 * SideStreams::kN); ++at) {
        std::set<cudaStream_t> used;
        g_calls = 0;
        g_fail_at = at;
        const int rc = build(&side, 8, false, &used);
        const bool reached = g_calls > at;
        g_fail_at = -1;
        need(!reached || rc, "a failed call was not reported");
        int open = 0;
        for (cudaStream_t s : used) open += g_seen[kCaller][s] < g_last[s];
        need(open <= 1, "one failed call left several streams unjoined");
    }
    std::set<cudaStream_t> used;
    need(build(nullptr, 3, false, &used) == 0 && used == std::set<cudaStream_t>{kCaller}, "no side streams: the caller's");
}

// Many handles: a bounded number of streams, given back with the last handle.
static void test_bounded() {
    std::vector<std::unique_ptr<StreamUser>> users;
    for (int i = 0; i < 512; ++i) {
        users.push_back(std::make_unique<StreamUser>());
        users.back()->attach(i % 2);
        std::set<cudaStream_t> used;
        need(build(users.back().get(), 10, false, &used) == 0, "build");
        need(used.size() == SideStreams::kN, "a build did not spread");
        need(g_streams <= 2 * StreamPool::kSets * SideStreams::kN, "streams grow with the handles");
    }
    users.clear();
    need(g_streams == 0 && g_events == 0, "the pool was not given back");
}

// Calls that are enqueuing at the same time hold different sets; past the
// last set a call runs on its own stream.
static void test_exclusive() {
    StreamUser u;
    u.attach(0);
    std::set<cudaStream_t> firsts;
    {
        std::vector<std::unique_ptr<Fork>> f;
        for (int i = 0; i < StreamPool::kSets + 1; ++i) {
            f.push_back(std::make_unique<Fork>(&u, kCaller));
            need(f.back()->begin() == cudaSuccess, "begin");
            need(firsts.insert(f.back()->at(0)).second, "one set lent twice");
        }
        need(f.back()->at(0) == kCaller && f.back()->at(3) == kCaller, "no set free: the caller's stream");
    }
    Fork again(&u, kCaller);
    need(again.begin() == cudaSuccess && again.at(0) != kCaller, "the sets were not given back");
    again.join();
    // threads
    std::vector<std::thread> t;
    std::map<cudaStream_t, int> busy;
    for (int i = 0; i < 8; ++i)
        t.emplace_back([&u, &busy, i] {
            for (int k = 0; k < 500; ++k) {
                Fork f(&u, (cudaStream_t)(uintptr_t)(0x100 + i));
                need(f.begin() == cudaSuccess, "begin");
                const cudaStream_t s = f.at(0);
                const bool own = s != (cudaStream_t)(uintptr_t)(0x100 + i);
                if (own) {
                    LOCKED;
                    need(busy[s]++ == 0, "two threads in one set");
                }
                std::this_thread::yield();
                if (own) {
                    LOCKED;
                    --busy[s];
                }
            }
        });
    for (auto &x : t) x.join();
}

// A set that a capture has joined is its own until the capture ends.
static void test_capture() {
    StreamUser u;
    u.attach(0);
    const cudaStream_t cs = (cudaStream_t)0x20;
    g_cap[cs] = 7;  // the first call is a captured one: it gets a set all the same
    const auto set_of = [&u](cudaStream_t st) {
        Fork f(&u, st);
        need(f.begin() == cudaSuccess, "begin");
        return f.at(0);
    };
    const cudaStream_t a = set_of(cs), b = set_of(cs);
    need(a != cs && a == b, "two builds in one capture");
    need(set_of(kCaller) != a, "a set lent out of a running capture");
    end_capture(7);
    need(set_of(kCaller) == a, "the capture's set comes back");
    need(!g_relaxed, "the capture mode was not put back");
}

// The side streams have the caller's priority.
static void test_priority() {
    StreamUser u;
    u.attach(0);
    const cudaStream_t high = (cudaStream_t)0x30;
    g_prio[high] = -5;
    for (cudaStream_t st : {kCaller, high, kCaller, high}) {
        Fork f(&u, st);
        need(f.begin() == cudaSuccess && f.at(0) != st, "begin");
        for (int i = 0; i < SideStreams::kN; ++i) need(g_prio[f.at(i)] == g_prio[st], "another priority than the caller's");
    }
}

int main() {
    test_joins();
    test_bounded();
    test_exclusive();
    test_capture();
    test_priority();
    need(g_streams == 0 && g_events == 0, "streams or events left");
    std::printf("ok\n");
}
