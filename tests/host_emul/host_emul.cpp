// host_emul.cpp -- host helpers of the library (csrc/cfg_sides.h) on a
// stand-in CUDA runtime that records every call and fails the one it is told to, for the
// tests: no GPU is involved, and no call fails on a real one.
#include "cfg_sides.h"

#include <cstdint>
#include <map>
#include <vector>

namespace {

enum Kind { LAUNCH, RECORD, WAIT, SYNC };
struct Op { Kind kind; const void* stream; const void* event; };
std::vector<Op> g_ops;
long g_calls = 0, g_fail_at = -1;   // calls that may fail so far; the one that does
uintptr_t g_next = 0x1000;

cudaError_t step() { return g_calls++ == g_fail_at ? cudaErrorUnknown : cudaSuccess; }

}  // namespace

extern "C" {

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) *s = (cudaStream_t)(g_next += 16);
    return e;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* ev, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) *ev = (cudaEvent_t)(g_next += 16);
    return e;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t s) {
    const cudaError_t e = step();
    if (e == cudaSuccess) g_ops.push_back(Op{RECORD, s, ev});
    return e;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t ev, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) g_ops.push_back(Op{WAIT, s, ev});
    return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { g_ops.push_back(Op{SYNC, s, nullptr}); return cudaSuccess; }

// One pass of `launches` launches in which call number fail_at fails (-1: none; the calls
// of create() are not counted).  -> 0: the pass kept its promise, else which one it broke;
// *calls: the calls that could have failed.
int side_streams_pass(uint32_t launches, long fail_at, long* calls) {
    using namespace cfg;
    g_fail_at = -1;
    SideStreams s;
    if (s.create() != cudaSuccess) return 1;
    const cudaStream_t main_stream = (cudaStream_t)(g_next += 16);
    g_ops.clear();
    g_calls = 0;
    g_fail_at = fail_at;
    cudaError_t e = s.fork(main_stream);
    if (e == cudaSuccess) {
        for (uint32_t t = 0; t < launches && e == cudaSuccess; ++t) {
            cudaStream_t on = nullptr;
            e = s.on(main_stream, t, on);
            if (e == cudaSuccess) e = step();   // the launch itself
            if (e == cudaSuccess) g_ops.push_back(Op{LAUNCH, on, nullptr});
        }
        const cudaError_t j = s.join(main_stream, e != cudaSuccess);
        if (e == cudaSuccess) e = j;
    }
    *calls = g_calls;
    g_fail_at = -1;
    if ((e == cudaSuccess) != (fail_at < 0 || fail_at >= g_calls)) return 2;   // an error that was lost, or made up
    std::map<const void*, size_t> first, last;
    for (size_t i = 0; i < g_ops.size(); ++i)
        if (g_ops[i].kind == LAUNCH) { first.emplace(g_ops[i].stream, i); last[g_ops[i].stream] = i; }
    for (const auto& [stream, at] : last) {
        bool waited = false, started = stream == main_stream, joined = stream == main_stream;
        for (size_t i = 0; i < g_ops.size(); ++i) {
            waited = waited || (i > at && g_ops[i].kind == SYNC && g_ops[i].stream == stream);
            started = started || (i < first[stream] && g_ops[i].kind == WAIT && g_ops[i].stream == stream &&
                                  g_ops[i].event == g_ops[0].event);
            if (i > at && g_ops[i].kind == RECORD && g_ops[i].stream == stream)
                for (size_t j = i + 1; j < g_ops.size(); ++j)
                    joined = joined || (g_ops[j].kind == WAIT && g_ops[j].stream == main_stream && g_ops[j].event == g_ops[i].event);
        }
        if (!started) return 3;                           // a launch that may overtake what main held at the fork
        if (e == cudaSuccess ? !joined : !waited) return 4;   // main runs on without it; the failed call returns before it ends
    }
    s.destroy();
    return 0;
}

}  // extern "C"
