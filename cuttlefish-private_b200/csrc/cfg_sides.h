// cfg_sides.h -- the launches of one pass spread over a stream and side streams of it.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace cfg {

// fork(main) opens a pass; its launch number t goes to the stream that on(main, t) gives:
// main itself or one of N side streams, each behind everything main held at the fork.
// join(main, failed) closes it: main goes behind every side stream used.  After an error --
// the pass's own (failed), or one in the join itself -- it waits on the host for main and
// for every side stream used instead: the buffers of a failed pass are free when it returns.
class SideStreams {
public:
    static constexpr uint32_t N = 3;

    // (a stream is made when a pass first has a launch for it: about 50 us each, an event 1 us)
    cudaError_t create() { return cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming); }
    void destroy() {
        for (uint32_t q = 0; q < N; ++q) {
            if (side_[q]) { cudaStreamSynchronize(side_[q]); cudaStreamDestroy(side_[q]); }
            if (join_[q]) cudaEventDestroy(join_[q]);
            side_[q] = nullptr; join_[q] = nullptr;
        }
        if (fork_) cudaEventDestroy(fork_);
        fork_ = nullptr;
    }

    cudaError_t fork(cudaStream_t main) {
        used_ = 0;
        return cudaEventRecord(fork_, main);
    }
    cudaError_t on(cudaStream_t main, uint32_t t, cudaStream_t& out) {
        const uint32_t q = t % (N + 1);
        cudaError_t e = cudaSuccess;
        if (q && !side_[q - 1]) e = cudaStreamCreateWithFlags(&side_[q - 1], cudaStreamNonBlocking);
        if (q && !join_[q - 1] && e == cudaSuccess) e = cudaEventCreateWithFlags(&join_[q - 1], cudaEventDisableTiming);
        out = q ? side_[q - 1] : main;
        if (!q || (used_ >> q & 1) || e != cudaSuccess) return e;
        e = cudaStreamWaitEvent(out, fork_, 0);
        if (e == cudaSuccess) used_ |= 1u << q;
        return e;
    }
    cudaError_t join(cudaStream_t main, bool failed) {
        cudaError_t e = cudaSuccess;
        for (uint32_t q = 1; q <= N && !failed && e == cudaSuccess; ++q) {
            if (!(used_ >> q & 1)) continue;
            e = cudaEventRecord(join_[q - 1], side_[q - 1]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(main, join_[q - 1], 0);
        }
        if (failed || e != cudaSuccess) {
            for (uint32_t q = 1; q <= N; ++q)
                if (used_ >> q & 1) cudaStreamSynchronize(side_[q - 1]);
            cudaStreamSynchronize(main);
        }
        used_ = 0;
        return e;
    }

private:
    cudaStream_t side_[N] = {};
    cudaEvent_t fork_ = nullptr, join_[N] = {};
    uint32_t used_ = 0;   // bit q: side stream q - 1 holds launches of this pass
};

}  // namespace cfg
