// host_emul.cpp -- host helpers of the library (csrc/cfg_sides.h, cfg_host.h) on a
// stand-in CUDA runtime that records every call and fails the one it is told to, for the
// tests: no GPU is involved, and no call fails on a real one.
#include "cfg_host.h"
#include "cfg_sides.h"

#include <cstdint>
#include <map>
#include <vector>

namespace {

enum Kind { LAUNCH, RECORD, WAIT, SYNC };
struct Op { Kind kind; const void* stream; const void* event; };
std::vector<Op> g_ops;
long g_calls = 0, g_fail_at = -1;   // calls that may fail so far; the one that does
long g_streams = 0;                 // made so far
uintptr_t g_next = 0x1000;

size_t g_room = SIZE_MAX, g_asked = 0;   // device bytes left to give out; bytes given out since the last reset
std::map<const void*, size_t> g_blocks;

cudaError_t step() { return g_calls++ == g_fail_at ? cudaErrorUnknown : cudaSuccess; }

}  // namespace

extern "C" {

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    const cudaError_t e = step();
    if (e == cudaSuccess) { *s = (cudaStream_t)(g_next += 16); ++g_streams; }
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

cudaError_t cudaMalloc(void** p, size_t n) {
    if (n > g_room) return cudaErrorMemoryAllocation;
    g_room -= n; g_asked += n;
    *p = (void*)(g_next += 256);   // never looked into
    g_blocks[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    g_room += g_blocks[p];
    g_blocks.erase(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t) { *p = (void*)(g_next += 256); return cudaSuccess; }
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }

// Collation buffers for n lm-tigs of k-mers of length k, twice with the device full after
// the first, then for `more` lm-tigs there is no room for.  -> 0, or the promise broken.
int unitig_buffers(uint64_t n, uint64_t more, uint32_t k) {
    cfg::UnitigBuffers ub;
    g_room = SIZE_MAX;
    if (!ub.ensure(n, k) || ub.held != n) return 1;
    g_room = 0;
    g_asked = 0;
    if (!ub.ensure(n, k) || g_asked) return 2;       // what is held is enough
    if (ub.held != n) return 3;
    if (ub.ensure(more, k) || ub.held != 0) return 4;   // a failed call lost a buffer, and says so
    g_room = SIZE_MAX;
    if (!ub.ensure(n, k) || ub.held != n) return 5;
    ub.release();
    return ub.held != 0 ? 6 : 0;
}

// Device bytes that the text parser's per-chunk state of `bytes` bytes of text asks for.
uint64_t parse_state_bytes(uint64_t bytes) {
    cfg::ParseBuffers pb;
    g_room = SIZE_MAX;
    g_asked = 0;
    const bool ok = pb.ensure_chunks((bytes + 4095) / 4096 + 1);
    pb.release();
    return ok ? g_asked : 0;
}

// Streams made by a SideStreams for a first pass of `launches` launches and a second one.
int side_streams_made(uint32_t launches) {
    cfg::SideStreams s;
    g_fail_at = -1;
    g_streams = 0;
    bool ok = s.create() == cudaSuccess && g_streams == 0;
    const cudaStream_t main_stream = (cudaStream_t)(g_next += 16);
    for (int pass = 0; pass < 2; ++pass) {
        ok = ok && s.fork(main_stream) == cudaSuccess;
        cudaStream_t on = nullptr;
        for (uint32_t t = 0; t < launches; ++t) ok = ok && s.on(main_stream, t, on) == cudaSuccess && on;
        ok = ok && s.join(main_stream, false) == cudaSuccess;
    }
    s.destroy();
    return ok ? (int)g_streams : -1;
}

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
