// cfg_partition.cu -- K1: weak super k-mer partitioning and bucket scatter.
//
// Restates Graph_Partitioner::process_chunk (src/Graph_Partitioner.cpp:505-597)
// with Min_Iterator<k-1> (include/Minimizer_Iterator.hpp:306-378) as a
// data-parallel sweep.  For every (k-1)-mer j of a fragment the subgraph is
// g_j = (min over its k-l l-mers of min(wyhash(l-mer), wyhash(rc(l-mer)))) & (G-1).
// The sequential cut rule (cut where g changes, or where the super (k-1)-mer
// reaches 2(k-1)-l bases) is equivalent to: pieces start at every g change and
// then every k-l (k-1)-mers inside a run of equal g.  So a run's pieces depend
// only on where the run starts, and a warp can own every run that starts in its
// stream segment, continuing past the segment's end until that run ends.
#include "cfg_device.cuh"
#include "cfg_internal.h"

#include <algorithm>

namespace cfg {

namespace {

constexpr int WARPS_PER_BLOCK = 8;
constexpr uint32_t STAGE = 256;       // records a warp gathers in shared memory per reservation

__device__ __forceinline__ uint32_t lanemask_lt() { uint32_t m; asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m)); return m; }

// A lane's l-mers of one fragment, one every 32 positions: min(hash(l-mer), hash(its reverse
// complement)), Min_Iterator::lmer_hash (include/Minimizer_Iterator.hpp:291-296).  A step moves
// the lane by one packed word and leaves its bit offsets as they are, so addresses and shifts
// are worked out once per fragment: this kernel is bound by the integer ALU pipe, not by loads
// (300 Mbp at k = 31, 3.56 -> 3.43 ms against working them out per l-mer; 150-base reads 3.89
// -> 3.82, 101-base reads at k = 27 1.49 -> 1.39 per 101 Mbp; k = 63 the same).
// With the reverse-complemented words at hand, the reverse complement is a second window: its
// first base is the l-mer's last, e = p + l - 1, at index 31 - (e mod 32) of rcw[e / 32], and it
// continues into rcw[e / 32 - 1].  Both windows always read their second word, the padding
// word after the stream's last (before rcw's first) where the l-mer needs no bit of it; a
// lane whose l-mer lies outside the fragment reads nothing and gets "none", all ones.
struct LmerWalk {
    const uint64_t *f, *r;    // the word of the l-mer's first base; of rcw, of its last
    uint32_t sf, sr;          // bits before the l-mer in its word; before its reverse complement in rcw's
    __device__ __forceinline__ LmerWalk(const PartitionArgs& a, int64_t p) {
        f = a.packed + (p >> 5); sf = 2 * (uint32_t)(p & 31);
        const int64_t e = p + a.l - 1;
        r = a.rcw + (e >> 5); sr = 62 - 2 * (uint32_t)(e & 31);
    }
    __device__ __forceinline__ uint64_t next(const PartitionArgs& a, bool valid) {
        uint64_t h = ~0ull;
        if (valid) {
            const uint32_t top = 64 - 2 * a.l;
            const uint64_t fw = ((__ldg(f) << sf) | ((__ldg(f + 1) >> 1) >> (63 - sf))) >> top;
            const uint64_t rc = a.rcw ? ((__ldg(r) << sr) | ((__ldg(r - 1) >> 1) >> (63 - sr))) >> top
                                      : rc_word(fw, a.l);
            const uint64_t x = wyhash8(fw, a.seed0), y = wyhash8(rc, a.seed0);
            h = x < y ? x : y;
        }
        ++f; ++r;
        return h;
    }
};

__global__ void k_rc_words(const uint64_t* __restrict__ packed, uint64_t w0, uint64_t w1, uint64_t* rcw) {
    for (uint64_t w = w0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < w1; w += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t r = __brevll(packed[w]);                                             // bits reversed
        r = ((r >> 1) & 0x5555555555555555ull) | ((r & 0x5555555555555555ull) << 1);  // each base's two bits restored
        rcw[w] = ~r;                                                                  // complemented: b -> 3 - b
    }
}

// A warp's records wait in shared memory and are reserved in the flat array together:
// one atomic on the run's record cursor per STAGE records instead of one per 32 positions.
struct Stage { uint64_t* buf; uint32_t n; };
__device__ __forceinline__ void stage_flush(const PartitionArgs& a, Stage& st) {
    if (st.n == 0) return;
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long b0 = 0;
    if (lane == 0) b0 = atomicAdd(a.rec_cursor, (unsigned long long)st.n);
    b0 = __shfl_sync(0xffffffffu, b0, 0);
    __syncwarp();
    for (uint32_t i = lane; i < st.n; i += 32) {
        const unsigned long long idx = b0 + i;
        if (idx < a.rec_cap) a.recs[idx] = st.buf[i]; else atomicOr(a.err, DERR_REC_OVERFLOW);
    }
    __syncwarp();
    st.n = 0;
}

// The value lane (lane - d) holds in this chunk, or for lanes < d the value lane
// (lane - d + 32) held in the previous chunk (0 <= d <= 31): each source lane supplies
// exactly one of the two, so one shuffle serves both.
__device__ __forceinline__ uint64_t from_back(uint64_t cur, uint64_t prev, uint32_t d, uint32_t lane) {
    return __shfl_sync(0xffffffffu, lane >= 32 - d ? prev : cur, (lane - d) & 31);
}
__device__ __forceinline__ uint64_t min64(uint64_t a, uint64_t b) { return a < b ? a : b; }

// The sparse table's depth E = floor(log2 w) is a template argument: levels 2^0 .. 2^E,
// none more (w = k - l <= 126: E <= 6).

// Processes the (k-1)-mer positions [j0, j1) of one fragment: emits every weak
// super k-mer whose run starts there.
// hist: this fragment's job's histogram (the run's, or its job's slice of a batch's);
// nullptr when the bucket sort counts the records itself.
//
// Window minima with warp shuffles: in the chunk of (k-1)-mers base .. base+31, lane L
// holds the newest l-mer hash, at q = base + w - 1 + L.  Level i of a sparse table holds
// at position q - 2^i + 1 the minimum of the 2^i hashes starting there: the minimum of
// the lane's own level i-1 value and that of the lane 2^(i-1) before it (for the first
// lanes, from the previous chunk).  The window of (k-1)-mer j = q - w + 1 is then two
// overlapping blocks of 2^E hashes, E = floor(log2 w): min(level_E[j], level_E[q-2^E+1]),
// the second the lane's own value, the first that of the lane w - 2^E before it.
// O(log w) work per position, no shared memory.  For w >= 96 (E = 6, dq = w - 64 > 32)
// the second block starts two chunks back: level E of the chunk before the previous is kept.
template <int E>
__device__ void sweep_fragment(const PartitionArgs& a, uint64_t F0, uint32_t FL, uint32_t j0, uint32_t j1,
                               unsigned long long* hist, Stage& st) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = a.k, l = a.l, w = a.w;
    const uint32_t M = FL - k + 2;                 // (k-1)-mers in the fragment
    const uint32_t n_lmers = FL - l + 1;
    const uint32_t start = j0 == 0 ? 0 : j0 - 1;   // position j0-1 only primes the change test
    const uint32_t dq = w - (1u << E);
    uint64_t lv[E + 1], pv[E + 1];   // this chunk's / the previous chunk's level values
    uint64_t ppE = ~0ull;            // level E two chunks back (E = 6 only)
#pragma unroll
    for (int i = 0; i <= E; ++i) pv[i] = ~0ull;
    auto levels = [&](uint64_t h) -> uint64_t {   // adds this chunk's hashes; the window minimum
        lv[0] = h;
#pragma unroll
        for (int i = 1; i <= E; ++i) lv[i] = min64(lv[i - 1], from_back(lv[i - 1], pv[i - 1], 1u << (i - 1), lane));
        uint64_t m;
        if constexpr (E >= 6) {   // dq <= 63: the block's start lies in one of the two chunks before
            m = dq <= 32 ? min64(lv[E], from_back(lv[E], pv[E], dq, lane))
                         : min64(lv[E], from_back(pv[E], ppE, dq - 32, lane));
            ppE = pv[E];
        } else {
            m = min64(lv[E], from_back(lv[E], pv[E], dq, lane));
        }
#pragma unroll
        for (int i = 0; i <= E; ++i) pv[i] = lv[i];
        return m;
    };
    // prime the levels with the chunks before the first: their hashes reach back to l-mer
    // `start`, ceil((w - 1) / 32) chunks (at least one)
    const int n_prime = (int)max(1u, (w - 1 + 31) / 32);
    const int64_t q0 = (int64_t)start + w - 1 + lane;   // the lane's l-mer in the first chunk
    LmerWalk lm(a, (int64_t)F0 + q0 - 32 * n_prime);
    for (int c = n_prime; c >= 1; --c) levels(lm.next(a, (uint64_t)(q0 - 32 * c) < (uint64_t)n_lmers));
    uint32_t left = q0 < (int64_t)n_lmers ? (uint32_t)(n_lmers - q0) : 0u;   // l-mers from the lane's next one to the end

    // Every change of g is a cut, so from a cut to the next one g is the same: a piece's g is that
    // of the position before the cut that ends it, and its start's "change" bit is in the mask.
    bool active = false;
    uint32_t last_cut = 0, last_cut_chg = 0;
    uint32_t carry_g = ~0u;   // g of the position before base (none at the fragment's start: a change)
    uint32_t carry_d = 0;     // base - start of the run in progress
    const uint32_t lt = lanemask_lt(), inside = min(M, j1);

    // each chunk's new l-mer hash is computed one chunk ahead, so its loads and
    // multiplies overlap the window minima of the chunk before
    uint64_t h_next = lm.next(a, left > 0);
    for (uint32_t base = start;; base += 32) {
        const uint64_t h = h_next;
        left = left > 32 ? left - 32 : 0u;
        h_next = lm.next(a, left > 0);
        const uint64_t m = levels(h);
        const uint32_t j = base + lane;
        const bool interior = base >= j0 && base + 32 <= inside;   // uniform: every position is one of [j0, j1)
        uint32_t g = (uint32_t)m & a.gmask;
        if (!interior && j >= M) g = 0;
        uint32_t gprev = __shfl_up_sync(0xffffffffu, g, 1);
        if (lane == 0) gprev = carry_g;
        const bool is_chg = gprev != g && (interior || (j < M && j >= j0));
        const uint32_t chg = __ballot_sync(0xffffffffu, is_chg);

        uint32_t act = 0xffffffffu, first = 0;   // positions of runs that start in [j0, j1); the first run's start
        if (!active) {
            if (chg == 0) {
                if (base + 32 >= j1 || base + 32 >= M) return;   // no run starts in [j0, j1)
                carry_g = __shfl_sync(0xffffffffu, g, 31);
                continue;
            }
            const uint32_t r0_lane = __ffs(chg) - 1;
            if (base + r0_lane >= j1) return;
            active = true;
            first = 1u << r0_lane;
            act = 0xffffffffu << r0_lane;
            last_cut = base + r0_lane;
            last_cut_chg = 1;
        }

        // distance to the start of the position's run: from the highest change at or below it,
        // else carried; a run is cut again every w positions, which a minimizer seldom reaches
        const uint32_t le = chg & (lt | (1u << lane));
        const uint32_t d = le ? lane - (31 - __clz(le)) : carry_d + lane;
        uint32_t cut = chg & act;
        if (__any_sync(0xffffffffu, d >= w && ((act >> lane) & 1)))
            cut = __ballot_sync(0xffffffffu, ((act >> lane) & 1) && (interior || j < M) && d % w == 0);

        // stop at the first change at or past j1: the run it starts belongs to the next segment
        bool stopping = false;
        if (base + 32 > j1) {
            const uint32_t stop = chg & __ballot_sync(0xffffffffu, j >= j1);   // (a change is a valid position)
            if (stop) {
                const uint32_t sl = __ffs(stop) - 1;
                cut &= (sl == 31) ? 0xffffffffu : ((2u << sl) - 1);
                stopping = true;
            }
        }
        const uint32_t emit = cut & ~first;   // piece [c, c') ends at every emitting lane c' = j
        const bool fin = !stopping && (base + 32 >= M);      // the fragment's last (k-1)-mer is in this chunk
        const uint32_t n_emit = __popc(emit) + (fin ? 1 : 0);
        if (st.n + n_emit > STAGE) stage_flush(a, st);
        const uint32_t slot0 = st.n;
        st.n += n_emit;
        if ((emit >> lane) & 1) {
            const uint32_t below = cut & lt, pl = 31 - __clz(below);
            const uint32_t c = below ? base + pl : last_cut;
            const uint32_t cchg = below ? (chg >> pl) & 1u : last_cut_chg;
            const uint32_t lj = c > 0;
            const uint32_t len = lj + (j - c + k - 2) + 1;
            const uint64_t r = rec_pack((uint32_t)(F0 + c - lj), len, lj & cchg, is_chg ? 1u : 0u, gprev);
            st.buf[slot0 + __popc(emit & lt)] = r;
            if (hist) atomicAdd(hist + gprev, 1ull | ((unsigned long long)(len - k + 1) << 32));
        }
        // carries: last cut / run start of this chunk
        if (cut) {
            const uint32_t hl = 31 - __clz(cut);
            last_cut = base + hl;
            last_cut_chg = (chg >> hl) & 1u;
        }
        if (fin) {   // final piece [last_cut, M): not joined on the right
            const uint32_t gl = __shfl_sync(0xffffffffu, g, M - 1 - base);
            if (lane == 0) {
                const uint32_t c = last_cut, lj = c > 0;
                const uint32_t len = lj + (FL - c);
                const uint64_t r = rec_pack((uint32_t)(F0 + c - lj), len, lj & last_cut_chg, 0, gl);
                st.buf[slot0 + __popc(emit)] = r;
                if (hist) atomicAdd(hist + gl, 1ull | ((unsigned long long)(len - k + 1) << 32));
            }
        }
        if (stopping || fin) return;
        carry_d = chg ? 32 - (31 - __clz(chg)) : carry_d + 32;
        carry_g = __shfl_sync(0xffffffffu, g, 31);
    }
}

// Four CTAs per SM (64 registers) for 32 <= w < 64, where the compiler's own choice is 96
// registers and two CTAs: 300 Mbp at k = 63 4.49 -> 3.98 ms.  The other depths are faster left
// at their 62 to 80 registers, three CTAs (k = 31: 3.43 ms at three CTAs; at 64 registers it lost 4 %).
template <int E>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32, E == 5 ? 4 : 0) k_partition(const PartitionArgs a) {
    __shared__ uint64_t stages[WARPS_PER_BLOCK][STAGE];
    Stage st{stages[threadIdx.x >> 5], 0};
    // this launch's bases and fragments (the fragment table is read only inside them:
    // the entries of other pieces may not have landed yet)
    const uint64_t b0 = a.base1 ? a.base0 : 0, b1 = a.base1 ? a.base1 : a.n_bases;
    const uint64_t f_lo = a.base1 ? a.frag_lo : 0, f_hi = a.base1 ? a.frag_hi : a.n_frags;
    const uint64_t n_seg = (b1 - b0 + a.seg - 1) / a.seg;
    const uint64_t warp0 = (uint64_t)blockIdx.x * WARPS_PER_BLOCK + (threadIdx.x >> 5);
    const uint64_t n_warps = (uint64_t)gridDim.x * WARPS_PER_BLOCK;
    for (uint64_t sgi = warp0; sgi < n_seg; sgi += n_warps) {
        const uint64_t s0 = b0 + sgi * a.seg, s1 = min(s0 + a.seg, b1);
        // last fragment starting at or before s0
        uint64_t lo = f_lo, hi = f_hi;
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) >> 1;
            if (a.frag_off[mid] <= s0) lo = mid; else hi = mid;
        }
        for (uint64_t f = lo; f < f_hi; ++f) {
            const uint64_t F0 = a.frag_off[f];
            if (F0 >= s1) break;
            const uint32_t FL = a.frag_len[f];
            // a device-resident fragment table is not checked on the host: a fragment past
            // the input or too short for a (k+1)-mer is skipped and reported
            if (FL < a.k + 1 || F0 + FL > a.n_bases) {
                if ((threadIdx.x & 31) == 0) atomicOr(a.err, DERR_BAD_FRAG);
                continue;
            }
            const uint32_t M = FL - a.k + 2;
            const uint32_t j0 = s0 > F0 ? (uint32_t)(s0 - F0) : 0;
            const uint64_t e = s1 - F0;
            const uint32_t j1 = e < M ? (uint32_t)e : M;
            if (j0 < j1) sweep_fragment<E>(a, F0, FL, j0, j1,
                                          a.hist ? a.hist + (a.frag_gbase ? a.frag_gbase[f] : 0u) : nullptr, st);
        }
    }
    stage_flush(a, st);
}

// Multi-block scans take 8192 entries per block.
constexpr uint32_t SCAN_PER_THREAD = 8, SCAN_BLOCK = 1024, SCAN_CHUNK = SCAN_PER_THREAD * SCAN_BLOCK;

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= (uint32_t)d) w += y;
        }
        warp_sums[lane] = w;   // inclusive
    }
    __syncthreads();
    total = warp_sums[(blockDim.x >> 5) - 1];
    const uint32_t before = wid ? warp_sums[wid - 1] : 0;
    __syncthreads();
    return before + x - v;
}

// Exclusive scan of the per-subgraph record counts by one block, 8192 entries at a time: a
// thread's 8 entries are 64 consecutive bytes (whole sectors), read with 16-byte loads and
// kept in registers between the sum and the write, so the histogram is read once.  Latency
// bound: 16384 subgraphs take 6 us where one pass of 16 strided entries a thread, a
// ten-barrier scan and a second read of the histogram took 44 us.
__global__ void __launch_bounds__(SCAN_BLOCK) k_bucket_scan(const unsigned long long* __restrict__ hist, uint32_t G,
                                                            uint32_t* bucket_off, uint32_t* inst, uint32_t* fill) {
    __shared__ uint32_t ws[32];
    uint32_t run0 = 0;
    for (uint32_t t0 = 0; t0 < G; t0 += SCAN_CHUNK) {
        const uint32_t b0 = t0 + threadIdx.x * SCAN_PER_THREAD;
        unsigned long long h[SCAN_PER_THREAD];
        const bool whole = b0 + SCAN_PER_THREAD <= G;
#pragma unroll
        for (uint32_t i = 0; i < SCAN_PER_THREAD; i += 2) {
            if (whole) {
                const ulonglong2 v = *(const ulonglong2*)(hist + b0 + i);
                h[i] = v.x; h[i + 1] = v.y;
            } else {
                h[i] = b0 + i < G ? hist[b0 + i] : 0ull;
                h[i + 1] = b0 + i + 1 < G ? hist[b0 + i + 1] : 0ull;
            }
        }
        uint32_t sum = 0, total;
#pragma unroll
        for (uint32_t i = 0; i < SCAN_PER_THREAD; ++i) sum += (uint32_t)h[i];
        uint32_t run = run0 + block_excl_scan(sum, ws, total);
#pragma unroll
        for (uint32_t i = 0; i < SCAN_PER_THREAD; ++i) {
            if (b0 + i >= G) break;
            bucket_off[b0 + i] = run;
            inst[b0 + i] = (uint32_t)(h[i] >> 32);
            fill[b0 + i] = 0;
            run += (uint32_t)h[i];
        }
        run0 += total;
    }
    if (threadIdx.x == 0) bucket_off[G] = run0;
}

// Multi-block scan for batches (millions of buckets).
__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_reduce(const unsigned long long* __restrict__ hist, uint32_t n,
                                                            uint32_t* partials) {
    __shared__ uint32_t ws[32];
    const uint64_t b0 = (uint64_t)blockIdx.x * SCAN_CHUNK + (uint64_t)threadIdx.x * SCAN_PER_THREAD;
    uint32_t sum = 0;
    for (uint32_t i = 0; i < SCAN_PER_THREAD; ++i)
        if (b0 + i < n) sum += (uint32_t)hist[b0 + i];
    uint32_t total;
    block_excl_scan(sum, ws, total);
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_partials(uint32_t* partials, uint32_t np) {
    __shared__ uint32_t ws[32];
    const uint32_t per = (np + SCAN_BLOCK - 1) / SCAN_BLOCK;
    const uint32_t p0 = threadIdx.x * per;
    uint32_t sum = 0;
    for (uint32_t i = 0; i < per; ++i)
        if (p0 + i < np) sum += partials[p0 + i];
    uint32_t total;
    uint32_t run = block_excl_scan(sum, ws, total);
    for (uint32_t i = 0; i < per; ++i)
        if (p0 + i < np) { const uint32_t v = partials[p0 + i]; partials[p0 + i] = run; run += v; }
}

__global__ void __launch_bounds__(SCAN_BLOCK) k_scan_apply(const unsigned long long* __restrict__ hist, uint32_t n,
                                                           const uint32_t* __restrict__ partials, uint32_t* bucket_off,
                                                           uint32_t* inst, uint32_t* fill) {
    __shared__ uint32_t ws[32];
    const uint64_t b0 = (uint64_t)blockIdx.x * SCAN_CHUNK + (uint64_t)threadIdx.x * SCAN_PER_THREAD;
    unsigned long long h[SCAN_PER_THREAD];
    uint32_t sum = 0;
    for (uint32_t i = 0; i < SCAN_PER_THREAD; ++i) {
        h[i] = b0 + i < n ? hist[b0 + i] : 0ull;
        sum += (uint32_t)h[i];
    }
    uint32_t total;
    uint32_t run = partials[blockIdx.x] + block_excl_scan(sum, ws, total);
    for (uint32_t i = 0; i < SCAN_PER_THREAD; ++i) {
        if (b0 + i >= n) break;
        bucket_off[b0 + i] = run;
        inst[b0 + i] = (uint32_t)(h[i] >> 32);
        fill[b0 + i] = 0;
        run += (uint32_t)h[i];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) bucket_off[n] = partials[blockIdx.x] + total;
}

__global__ void k_scatter(const ScatterArgs a) {
    const uint64_t n = a.n_dev ? *a.n_dev : a.n;
    if (n > a.n) return;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = a.flat[i];
        uint32_t g = rec_g(r);
        if (a.job_pos) {   // the record's job: the last job starting at or before its first base
            const uint64_t p = rec_pos(r);
            uint32_t lo = 0, hi = a.n_jobs;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (a.job_pos[mid] <= p) lo = mid; else hi = mid;
            }
            g += lo << a.g_shift;
        }
        const uint32_t slot = atomicAdd(a.bucket_fill + g, 1u);
        a.recs[a.bucket_off[g] + slot] = r;
    }
}

}  // namespace

void launch_partition(const PartitionArgs& a, cudaStream_t s) {
    const uint64_t n_seg = ((a.base1 ? a.base1 - a.base0 : a.n_bases) + a.seg - 1) / a.seg;
    uint64_t blocks = (n_seg + WARPS_PER_BLOCK - 1) / WARPS_PER_BLOCK;
    if (blocks > (1u << 20)) blocks = 1u << 20;
    if (blocks == 0) return;
    const dim3 grid((unsigned)blocks), block(WARPS_PER_BLOCK * 32);
    switch (31 - __builtin_clz(a.w)) {   // floor(log2 w), w = k - l in [1, 126]
        case 0: k_partition<0><<<grid, block, 0, s>>>(a); break;
        case 1: k_partition<1><<<grid, block, 0, s>>>(a); break;
        case 2: k_partition<2><<<grid, block, 0, s>>>(a); break;
        case 3: k_partition<3><<<grid, block, 0, s>>>(a); break;
        case 4: k_partition<4><<<grid, block, 0, s>>>(a); break;
        case 5: k_partition<5><<<grid, block, 0, s>>>(a); break;
        default: k_partition<6><<<grid, block, 0, s>>>(a); break;
    }
}

void launch_rc_words(const uint64_t* packed, uint64_t w0, uint64_t w1, uint64_t* rcw, cudaStream_t s) {
    if (w1 <= w0) return;
    const uint64_t blocks = std::min<uint64_t>((w1 - w0 + 255) / 256, 148ull * 16);
    k_rc_words<<<(unsigned)blocks, 256, 0, s>>>(packed, w0, w1, rcw);
}

void launch_bucket_scan(const unsigned long long* hist, uint32_t G, uint32_t* bucket_off, uint32_t* inst,
                        uint32_t* fill, cudaStream_t s) {
    k_bucket_scan<<<1, SCAN_BLOCK, 0, s>>>(hist, G, bucket_off, inst, fill);
}

void launch_bucket_scan_large(const unsigned long long* hist, uint32_t n, uint32_t* bucket_off, uint32_t* inst,
                              uint32_t* fill, uint32_t* partials, cudaStream_t s) {
    const uint32_t nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
    k_scan_reduce<<<nb, SCAN_BLOCK, 0, s>>>(hist, n, partials);
    k_scan_partials<<<1, SCAN_BLOCK, 0, s>>>(partials, nb);
    k_scan_apply<<<nb, SCAN_BLOCK, 0, s>>>(hist, n, partials, bucket_off, inst, fill);
}

void launch_scatter(const ScatterArgs& a, cudaStream_t s) {
    if (a.n == 0) return;
    uint64_t blocks = (a.n + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    k_scatter<<<(unsigned)blocks, 256, 0, s>>>(a);
}

}  // namespace cfg
