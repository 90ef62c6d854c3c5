// The stream fork (side_streams.h) on the CPU: the CUDA calls it makes are
// counted by the stand-ins below instead of the runtime.  Prints "ok" or the
// first thing that is wrong; built and run by tests/test_side_streams.py.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <set>
#include <vector>

#include "side_streams.h"

using namespace fjb;

// what the stand-in runtime saw
static int g_streams, g_events, g_launches;          // live streams and events, launches so far
static std::map<cudaStream_t, int> g_last;           // a stream's last launch
static std::map<cudaEvent_t, std::map<cudaStream_t, int>> g_event;  // what an event covers
static std::map<cudaStream_t, std::map<cudaStream_t, int>> g_seen;  // what a stream has waited for
static int g_fail_at = -1, g_calls;                  // the call that fails, if any

static cudaError_t call() { return g_calls++ == g_fail_at ? cudaErrorUnknown : cudaSuccess; }
static void need(bool ok, const char *what) {
    if (ok) return;
    std::printf("%s\n", what);
    std::exit(1);
}

extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = (cudaStream_t)std::malloc(1);
    ++g_streams;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    --g_streams;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    *e = (cudaEvent_t)std::malloc(1);
    ++g_events;
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    --g_events;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (cudaError_t r = call()) return r;
    g_event[e] = g_seen[s];
    g_event[e][s] = g_last[s];
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (cudaError_t r = call()) return r;
    for (auto &kv : g_event[e])
        if (kv.second > g_seen[s][kv.first]) g_seen[s][kv.first] = kv.second;
    return cudaSuccess;
}
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
static int build(SideStreams *side, int n, bool early, std::set<cudaStream_t> *used) {
    Fork fork(side, kCaller);
    if (fork.begin() != cudaSuccess) return 1;
    for (int i = 0; i < n; ++i) {
        used->insert(fork.at(i));
        launch(fork.at(i));
    }
    if (early) return 1;
    return fork.join() != cudaSuccess;
}

static void test_joins() {
    SideStreams side;
    need(side.ensure() == cudaSuccess, "ensure");
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

int main() {
    test_joins();
    need(g_streams == 0 && g_events == 0, "streams or events left");
    std::printf("ok\n");
}
