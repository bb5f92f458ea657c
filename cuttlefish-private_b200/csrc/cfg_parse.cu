// cfg_parse.cu -- FASTA / FASTQ text to the packed input, on the device.
//
// The input side of Graph_Partitioner (record parsing by RabbitFX,
// include/RabbitFX/io/Formater.cpp:87-130,265-297, and the fragment scan of
// process_chunk, src/Graph_Partitioner.cpp:461-501) as data-parallel passes over
// the raw text in HBM.  A FASTA record's sequence is its lines joined; a FASTQ
// record's is its second line.  Fragments are the maximal runs of ACGT (either
// case) inside a record's sequence; those shorter than k+1 bases are dropped.
//
// Every byte is read by a finite-state machine (the line structure of the
// format) that gives the byte a class: skipped (header, quality, newline),
// a base, or a break (a non-ACGT character, a record boundary).  The state at
// each 4 KiB chunk is found by composing the chunks' state-transfer functions
// (a scan), so every chunk runs independently:
//   A  transfer function of every chunk (and of every group's bytes before it, kept
//      for C)                                       B  scan: each chunk's start state
//   C  each group's emissions as two 16-bit masks (kept for E and G, in the word that held
//      A's function), bases and breaks of the chunk and before every 32 of its groups
//                                                   D  scan: each chunk's offsets
//   E  the base rank of every break                F  fragments: lengths, keep, offsets
//   G  bases written 2 bits each into the packed stream.
// A and C give a warp a whole chunk, 32 groups of 16 bytes at a time: no barrier, every
// load of the chunk in flight at once, the scan carried in registers.  E and G visit only
// the groups with breaks, or bases, to place, and find what is before a group by a scan over
// the warp: 4 bytes per group and 4 per 32 groups are all that is kept, 0.26 bytes per byte of
// text (a prefix and the masks of every group, in words of their own beside A's function: 0.63
// bytes, and 1.74 ms where this takes 1.63; with one group to a lane the scans made it 1.81).
// What is done with a group's 16 bytes is in cfg_parse_thread.cuh.  Bound: instruction issue
// (the text is read three times, 0.3 ms of the 1.63 ms that 630 MB of FASTQ take; 8.8 ms with a
// byte-by-byte walk of the groups that hold a newline, CTA-wide scans and one-CTA scans over
// the chunks).
#include "cuttlefish_gpu.h"
#include "cfg_host.h"
#include "cfg_internal.h"
#include "cfg_parse_thread.cuh"

#include <algorithm>

namespace cfg {

namespace {

using namespace parse;

struct ParseArgs {
    const uint8_t* text;
    uint64_t bytes, n_chunks;
    FsmBits fsm;
    uint32_t* chunk_f;             // A: transfer function; B: start state
    uint32_t* group_w;             // A: per group, the chunk's function before it; C: its bytes that are bases (low
                                   // half) and breaks (high half)
    uint32_t* step_pre;            // C: per 32 groups, the chunk's bases and breaks before them
    uint32_t* part_f;              // B: transfer function of every 1024 chunks
    unsigned long long* part_s;    // C: bases and breaks of every 1024 chunks
    unsigned long long* chunk_b;   // C: bases; D: bases before the chunk
    unsigned long long* chunk_k;   // C: breaks; D: breaks before the chunk
    unsigned long long* brk_rank;  // E: bases before break i (NB + 1 entries)
    uint64_t* packed;
    const unsigned long long* frag_out;   // F: output start of fragment i, ~0 if dropped
};

constexpr uint32_t FULL = 0xffffffffu;
constexpr uint32_t WARP_GROUPS = TPB / 32;   // groups a lane takes of its warp's chunk: 8
constexpr uint32_t SCAN_CHUNKS = 1024;       // chunks per CTA of the scans B and D

// The 16 bytes at p (zero past the end).
__device__ __forceinline__ Group load_group(const ParseArgs& a, uint64_t p) {
    Group g;
    if (p + BPT <= a.bytes) {
        const uint4 w = *(const uint4*)(a.text + p);
        g.w[0] = w.x; g.w[1] = w.y; g.w[2] = w.z; g.w[3] = w.w;
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t x = 0;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (p + 4 * j + i < a.bytes) x |= (uint32_t)a.text[p + 4 * j + i] << (8 * i);
            g.w[j] = x;
        }
    }
    return g;
}
__device__ __forceinline__ uint32_t bytes_at(const ParseArgs& a, uint64_t p) {   // of the group at p
    return p >= a.bytes ? 0 : (uint32_t)umin64(BPT, a.bytes - p);
}

__device__ __forceinline__ Fn identity_fn() { return Fn{0x03020100u, 4u}; }
__device__ __forceinline__ Fn shfl_fn(Fn f, int src) { return Fn{__shfl_sync(FULL, f.lo, src), __shfl_sync(FULL, f.hi, src)}; }
// Inclusive scan of transfer functions over the warp (in lane order).
__device__ __forceinline__ Fn warp_scan_fn(Fn x, uint32_t lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Fn y{__shfl_up_sync(FULL, x.lo, d), __shfl_up_sync(FULL, x.hi, d)};
        if (lane >= (uint32_t)d) x = fn_then(y, x);
    }
    return x;
}

// A: the chunk's transfer function.
__global__ void __launch_bounds__(TPB) k_parse_transfer(ParseArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (TPB / 32);
    for (uint64_t c = (uint64_t)blockIdx.x * (TPB / 32) + (threadIdx.x >> 5); c < a.n_chunks; c += nw) {
        Group g[WARP_GROUPS];
#pragma unroll
        for (uint32_t i = 0; i < WARP_GROUPS; ++i) g[i] = load_group(a, c * CHUNK + (uint64_t)(i * 32 + lane) * BPT);
        Fn carry = identity_fn();
#pragma unroll
        for (uint32_t i = 0; i < WARP_GROUPS; ++i) {
            const uint32_t t = i * 32 + lane;
            const Fn x = warp_scan_fn(thread_fn(a.fsm, g[i], bytes_at(a, c * CHUNK + (uint64_t)t * BPT)), lane);
            const Fn up{__shfl_up_sync(FULL, x.lo, 1), __shfl_up_sync(FULL, x.hi, 1)};
            a.group_w[c * TPB + t] = fn_bits(lane ? fn_then(carry, up) : carry);
            carry = fn_then(carry, shfl_fn(x, 31));
        }
        if (lane == 0) a.chunk_f[c] = fn_bits(carry);
    }
}

// The functions of the 4 chunks of this thread (of the CTA's SCAN_CHUNKS) composed, and
// the exclusive scan of those over the CTA; `all`: the CTA's whole function.
__device__ __forceinline__ Fn block_scan_fn(Fn f, Fn* sh, Fn& all) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const Fn x = warp_scan_fn(f, lane);
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    Fn before = identity_fn();
    all = identity_fn();
#pragma unroll
    for (uint32_t w = 0; w < TPB / 32; ++w) {
        if (w == wid) before = all;
        all = fn_then(all, sh[w]);
    }
    const Fn up{__shfl_up_sync(FULL, x.lo, 1), __shfl_up_sync(FULL, x.hi, 1)};
    __syncthreads();
    return lane ? fn_then(before, up) : before;
}
static_assert(SCAN_CHUNKS == 4 * TPB, "a thread takes 4 chunks");

// B, first pass: the transfer function of every SCAN_CHUNKS chunks.
__global__ void __launch_bounds__(TPB) k_parse_states_sum(ParseArgs a) {
    __shared__ Fn sh[TPB / 32];
    const uint64_t c0 = (uint64_t)blockIdx.x * SCAN_CHUNKS + 4 * threadIdx.x;
    Fn f = identity_fn(), all;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
        if (c0 + j < a.n_chunks) f = fn_then(f, fn_of(a.chunk_f[c0 + j]));
    block_scan_fn(f, sh, all);
    if (threadIdx.x == 0) a.part_f[blockIdx.x] = fn_bits(all);
}

// B, second pass: each chunk's start state.
__global__ void __launch_bounds__(TPB) k_parse_states(ParseArgs a) {
    __shared__ Fn sh[TPB / 32];
    // the CTAs before this one, a contiguous share per thread
    const uint32_t per = (blockIdx.x + TPB - 1) / TPB;
    const uint32_t p0 = min(blockIdx.x, threadIdx.x * per), p1 = min(blockIdx.x, p0 + per);
    Fn f = identity_fn(), base, all;
    for (uint32_t p = p0; p < p1; ++p) f = fn_then(f, fn_of(a.part_f[p]));
    block_scan_fn(f, sh, base);
    const uint64_t c0 = (uint64_t)blockIdx.x * SCAN_CHUNKS + 4 * threadIdx.x;
    uint32_t tf[4];
    f = identity_fn();
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        tf[j] = c0 + j < a.n_chunks ? a.chunk_f[c0 + j] : 0u;
        if (c0 + j < a.n_chunks) f = fn_then(f, fn_of(tf[j]));
    }
    const Fn ex = block_scan_fn(f, sh, all);
    uint32_t st = f_at(fn_bits(fn_then(base, ex)), a.fsm.start);
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
        if (c0 + j < a.n_chunks) {
            a.chunk_f[c0 + j] = st;
            st = f_at(tf[j], st);
        }
}

// C: emissions of every group, bases and breaks of every chunk, and before every group.
__global__ void __launch_bounds__(TPB) k_parse_counts(ParseArgs a) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = (uint64_t)gridDim.x * (TPB / 32);
    for (uint64_t c = (uint64_t)blockIdx.x * (TPB / 32) + (threadIdx.x >> 5); c < a.n_chunks; c += nw) {
        Group g[WARP_GROUPS];
        uint32_t tf[WARP_GROUPS];
#pragma unroll
        for (uint32_t i = 0; i < WARP_GROUPS; ++i) {
            g[i] = load_group(a, c * CHUNK + (uint64_t)(i * 32 + lane) * BPT);
            tf[i] = a.group_w[c * TPB + i * 32 + lane];
        }
        const uint32_t st = a.chunk_f[c];
        uint32_t carry = 0;   // bases | breaks << 16 before this step's groups (a chunk holds 4096 bytes)
#pragma unroll
        for (uint32_t i = 0; i < WARP_GROUPS; ++i) {
            const uint32_t t = i * 32 + lane;
            const Emits e = thread_emits(a.fsm, f_at(tf[i], st), g[i], bytes_at(a, c * CHUNK + (uint64_t)t * BPT));
            if (lane == 0) a.step_pre[c * WARP_GROUPS + i] = carry;
            a.group_w[c * TPB + t] = emits_word(e);
            carry += __reduce_add_sync(FULL, emits_counts(e));
        }
        if (lane == 0) {
            a.chunk_b[c] = pre_bases(carry); a.chunk_k[c] = pre_breaks(carry);
            unsigned long long* ps = a.part_s + 2 * (c / SCAN_CHUNKS);
            atomicAdd(ps, (unsigned long long)pre_bases(carry));
            atomicAdd(ps + 1, (unsigned long long)pre_breaks(carry));
        }
    }
}

// Exclusive scan over the CTA of two sums; their totals in tot.
__device__ __forceinline__ void block_scan2(unsigned long long& x, unsigned long long& y, unsigned long long (*sh)[2],
                                            unsigned long long (&tot)[2]) {
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long a = x, b = y;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long p = __shfl_up_sync(FULL, a, d), q = __shfl_up_sync(FULL, b, d);
        if (lane >= (uint32_t)d) { a += p; b += q; }
    }
    if (lane == 31) { sh[wid][0] = a; sh[wid][1] = b; }
    __syncthreads();
    unsigned long long ba = 0, bb = 0;
    tot[0] = tot[1] = 0;
#pragma unroll
    for (uint32_t w = 0; w < TPB / 32; ++w) {
        if (w == wid) { ba = tot[0]; bb = tot[1]; }
        tot[0] += sh[w][0]; tot[1] += sh[w][1];
    }
    __syncthreads();
    x = ba + a - x; y = bb + b - y;
}

// D: exclusive prefix sums of the chunks' bases and breaks; the last entries (index
// n_chunks) get the totals.
__global__ void __launch_bounds__(TPB) k_parse_offsets(ParseArgs a) {
    __shared__ unsigned long long sh[TPB / 32][2];
    unsigned long long b = 0, k = 0, base[2], tot[2];
    for (uint32_t p = threadIdx.x; p < blockIdx.x; p += TPB) { b += a.part_s[2 * p]; k += a.part_s[2 * p + 1]; }
    block_scan2(b, k, sh, base);
    const uint64_t c0 = (uint64_t)blockIdx.x * SCAN_CHUNKS + 4 * threadIdx.x;
    unsigned long long cb[4], ck[4];
    b = k = 0;
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) {
        cb[j] = c0 + j < a.n_chunks ? a.chunk_b[c0 + j] : 0ull;
        ck[j] = c0 + j < a.n_chunks ? a.chunk_k[c0 + j] : 0ull;
        b += cb[j]; k += ck[j];
    }
    block_scan2(b, k, sh, tot);
    b += base[0]; k += base[1];
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
        if (c0 + j < a.n_chunks) {
            a.chunk_b[c0 + j] = b; a.chunk_k[c0 + j] = k;
            b += cb[j]; k += ck[j];
        }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        a.chunk_b[a.n_chunks] = base[0] + tot[0];
        a.chunk_k[a.n_chunks] = base[1] + tot[1];
    }
}

// Bases and breaks of the chunk before the lane's groups: the warp's lanes hold `own` each, in
// order, and its first group starts step `step`.
__device__ __forceinline__ uint32_t groups_pre(const ParseArgs& a, uint64_t step, uint32_t own) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t x = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    return a.step_pre[step] + x - own;
}

// E: for every break, the number of bases before it; break NB (after the text) closes
// the last fragment.  Four groups to a lane, so that the warp's scan serves 128 of them;
// a warp runs whole, and within one chunk.
__global__ void __launch_bounds__(TPB) k_parse_breaks(ParseArgs a) {
    constexpr uint32_t N = 4;
    const uint64_t n = a.n_chunks * (TPB / N), stride = (uint64_t)gridDim.x * TPB;
    for (uint64_t i = (uint64_t)blockIdx.x * TPB + threadIdx.x; i < n; i += stride) {
        const uint4 m = ((const uint4*)a.group_w)[i];
        if (!__any_sync(FULL, (m.x | m.y | m.z | m.w) >> 16)) continue;
        const uint32_t w[N] = {m.x, m.y, m.z, m.w};
        uint32_t own = 0;
#pragma unroll
        for (uint32_t j = 0; j < N; ++j) own += emits_counts(word_emits(w[j]));
        uint32_t pre = groups_pre(a, (i / 32) * N, own);
        const unsigned long long r = a.chunk_b[i / (TPB / N)], kk = a.chunk_k[i / (TPB / N)];
#pragma unroll
        for (uint32_t j = 0; j < N; ++j) {
            const Emits e = word_emits(w[j]);
            emit_breaks(e, r + pre_bases(pre), kk + pre_breaks(pre), a.brk_rank);
            pre += emits_counts(e);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) a.brk_rank[a.chunk_k[a.n_chunks]] = a.chunk_b[a.n_chunks];
}

// F: fragment i holds the bases between breaks i-1 and i; kept if it has k+1 of
// them.  Three steps: keep flags and lengths, a scan, then the tables.
struct FragArgs {
    const unsigned long long* brk_rank;
    uint64_t n_frag;                    // breaks + 1
    uint32_t k;
    unsigned long long* out;            // per fragment: output start, ~0 if dropped
    uint32_t* part_n; unsigned long long* part_b;   // per block: kept fragments, kept bases
    uint64_t* frag_off; uint32_t* frag_len;
    unsigned long long* totals;         // [0] kept fragments, [1] kept bases
};

constexpr uint32_t FR_PER_BLOCK = 1024 * 4;

__device__ __forceinline__ uint64_t frag_len_at(const FragArgs& f, uint64_t i) {
    return f.brk_rank[i] - (i ? f.brk_rank[i - 1] : 0ull);
}

__global__ void __launch_bounds__(1024) k_frag_reduce(FragArgs f) {
    __shared__ unsigned long long sb[32];
    __shared__ uint32_t sn[32];
    const uint64_t i0 = (uint64_t)blockIdx.x * FR_PER_BLOCK + threadIdx.x * 4;
    uint32_t n = 0;
    unsigned long long b = 0;
    for (uint32_t j = 0; j < 4; ++j) {
        const uint64_t i = i0 + j;
        if (i >= f.n_frag) break;
        const uint64_t L = frag_len_at(f, i);
        if (L >= f.k + 1) { ++n; b += L; }
    }
    for (int d = 16; d; d >>= 1) { n += __shfl_down_sync(0xffffffffu, n, d); b += __shfl_down_sync(0xffffffffu, b, d); }
    if ((threadIdx.x & 31) == 0) { sn[threadIdx.x >> 5] = n; sb[threadIdx.x >> 5] = b; }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t tn = 0; unsigned long long tb = 0;
        for (int w = 0; w < 32; ++w) { tn += sn[w]; tb += sb[w]; }
        f.part_n[blockIdx.x] = tn; f.part_b[blockIdx.x] = tb;
    }
}

__global__ void __launch_bounds__(1024) k_frag_scan(FragArgs f, uint32_t nblocks) {
    __shared__ unsigned long long sb[1024];
    __shared__ uint32_t sn[1024];
    const uint32_t per = (nblocks + 1023) / 1024;
    const uint32_t p0 = min(nblocks, threadIdx.x * per), p1 = min(nblocks, p0 + per);
    uint32_t n = 0; unsigned long long b = 0;
    for (uint32_t p = p0; p < p1; ++p) { n += f.part_n[p]; b += f.part_b[p]; }
    sn[threadIdx.x] = n; sb[threadIdx.x] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t rn = 0; unsigned long long rb = 0;
        for (uint32_t t = 0; t < 1024; ++t) { const uint32_t x = sn[t]; const unsigned long long y = sb[t]; sn[t] = rn; sb[t] = rb; rn += x; rb += y; }
        f.totals[0] = rn; f.totals[1] = rb;
    }
    __syncthreads();
    uint32_t rn = sn[threadIdx.x]; unsigned long long rb = sb[threadIdx.x];
    for (uint32_t p = p0; p < p1; ++p) {
        const uint32_t x = f.part_n[p]; const unsigned long long y = f.part_b[p];
        f.part_n[p] = rn; f.part_b[p] = rb; rn += x; rb += y;
    }
}

__global__ void __launch_bounds__(1024) k_frag_write(FragArgs f) {
    __shared__ unsigned long long wb[32];
    __shared__ uint32_t wn[32];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t i0 = (uint64_t)blockIdx.x * FR_PER_BLOCK + threadIdx.x * 4;
    uint64_t L[4]; bool keep[4];
    uint32_t n = 0; unsigned long long b = 0;
    for (uint32_t j = 0; j < 4; ++j) {
        const uint64_t i = i0 + j;
        L[j] = i < f.n_frag ? frag_len_at(f, i) : 0;
        keep[j] = i < f.n_frag && L[j] >= f.k + 1;
        if (keep[j]) { ++n; b += L[j]; }
    }
    uint32_t xn = n; unsigned long long xb = b;   // inclusive warp scan
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t pn = __shfl_up_sync(0xffffffffu, xn, d);
        const unsigned long long pb = __shfl_up_sync(0xffffffffu, xb, d);
        if (lane >= (uint32_t)d) { xn += pn; xb += pb; }
    }
    if (lane == 31) { wn[wid] = xn; wb[wid] = xb; }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t rn = f.part_n[blockIdx.x]; unsigned long long rb = f.part_b[blockIdx.x];
        for (int w = 0; w < 32; ++w) { const uint32_t x = wn[w]; const unsigned long long y = wb[w]; wn[w] = rn; wb[w] = rb; rn += x; rb += y; }
    }
    __syncthreads();
    uint32_t idx = wn[wid] + xn - n;
    unsigned long long at = wb[wid] + xb - b;
    for (uint32_t j = 0; j < 4; ++j) {
        const uint64_t i = i0 + j;
        if (i >= f.n_frag) break;
        if (keep[j]) {
            f.out[i] = at;
            f.frag_off[idx] = at; f.frag_len[idx] = (uint32_t)L[j];
            ++idx; at += L[j];
        } else {
            f.out[i] = ~0ull;
        }
    }
}

struct AtomicOr64 {
    __device__ __forceinline__ void operator()(uint64_t* w, uint64_t bits) const {
        atomicOr((unsigned long long*)w, (unsigned long long)bits);
    }
};

// G: every kept base to its place in the packed stream (MSB-first, 32 per word).  Two
// groups to a lane (as in E); only groups that emit a base read their bytes.
__global__ void __launch_bounds__(TPB) k_parse_pack(ParseArgs a) {
    constexpr uint32_t N = 2;
    const uint64_t n = a.n_chunks * (TPB / N), stride = (uint64_t)gridDim.x * TPB;
    for (uint64_t i = (uint64_t)blockIdx.x * TPB + threadIdx.x; i < n; i += stride) {
        const uint2 m = ((const uint2*)a.group_w)[i];
        if (!__any_sync(FULL, (m.x | m.y) & 0xFFFFu)) continue;
        const uint32_t w[N] = {m.x, m.y};
        uint32_t pre = groups_pre(a, (i / 32) * N, emits_counts(word_emits(m.x)) + emits_counts(word_emits(m.y)));
        const unsigned long long r = a.chunk_b[i / (TPB / N)], kk = a.chunk_k[i / (TPB / N)];
#pragma unroll
        for (uint32_t j = 0; j < N; ++j) {
            const Emits e = word_emits(w[j]);
            if (e.base)
                emit_pack(e, load_group(a, (i * N + j) * BPT), r + pre_bases(pre), kk + pre_breaks(pre), a.frag_out,
                          a.brk_rank, a.packed, AtomicOr64{});
            pre += emits_counts(e);
        }
    }
}

}  // namespace

int parse_text_device(const uint8_t* d_text, uint64_t bytes, int fastq, uint32_t k, ParseBuffers& pb, cudaStream_t s) {
    ParseArgs a{};
    a.text = d_text; a.bytes = bytes;
    a.n_chunks = (bytes + CHUNK - 1) / CHUNK;
    a.fsm = pack_fsm(fastq ? fastq_fsm() : fasta_fsm());
    const uint64_t nc = a.n_chunks;
    if (!pb.ensure_chunks(nc + 1)) return CFG_ERR_OOM;
    a.chunk_f = pb.chunk_f; a.chunk_b = pb.chunk_b; a.chunk_k = pb.chunk_k;
    a.group_w = pb.group_w; a.step_pre = pb.step_pre; a.part_f = pb.chunk_part_f; a.part_s = pb.chunk_part_s;
    const unsigned wgrid = (unsigned)std::min<uint64_t>((nc + TPB / 32 - 1) / (TPB / 32), 148ull * 32);   // a warp per chunk
    const unsigned bgrid = (unsigned)std::min<uint64_t>((nc + 3) / 4, 148ull * 32), pgrid = (unsigned)std::min<uint64_t>((nc + 1) / 2, 148ull * 32);
    const unsigned sgrid = (unsigned)std::max<uint64_t>((nc + SCAN_CHUNKS - 1) / SCAN_CHUNKS, 1);
    if (cudaMemsetAsync(a.part_s, 0, 16ull * sgrid, s) != cudaSuccess) return CFG_ERR_CUDA;
    if (nc) {
        k_parse_transfer<<<wgrid, TPB, 0, s>>>(a);
        k_parse_states_sum<<<sgrid, TPB, 0, s>>>(a);
        k_parse_states<<<sgrid, TPB, 0, s>>>(a);
        k_parse_counts<<<wgrid, TPB, 0, s>>>(a);
    }
    k_parse_offsets<<<sgrid, TPB, 0, s>>>(a);
    unsigned long long tot[2] = {0, 0};   // bases, breaks
    if (cudaMemcpyAsync(&tot[0], a.chunk_b + nc, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaMemcpyAsync(&tot[1], a.chunk_k + nc, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return CFG_ERR_CUDA;
    const uint64_t n_frag = tot[1] + 1;
    if (!pb.ensure_frags(n_frag)) return CFG_ERR_OOM;
    a.brk_rank = pb.brk_rank;
    if (nc) k_parse_breaks<<<bgrid, TPB, 0, s>>>(a);
    else if (cudaMemsetAsync(a.brk_rank, 0, 8, s) != cudaSuccess) return CFG_ERR_CUDA;
    FragArgs f{};
    f.brk_rank = pb.brk_rank; f.n_frag = n_frag; f.k = k; f.out = pb.frag_out;
    f.part_n = pb.part_n; f.part_b = pb.part_b; f.frag_off = pb.frag_off; f.frag_len = pb.frag_len; f.totals = pb.totals;
    const uint32_t nfb = (uint32_t)((n_frag + FR_PER_BLOCK - 1) / FR_PER_BLOCK);
    k_frag_reduce<<<nfb, 1024, 0, s>>>(f);
    k_frag_scan<<<1, 1024, 0, s>>>(f, nfb);
    k_frag_write<<<nfb, 1024, 0, s>>>(f);
    unsigned long long kept[2] = {0, 0};
    if (cudaMemcpyAsync(kept, pb.totals, 16, cudaMemcpyDeviceToHost, s) != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
        return CFG_ERR_CUDA;
    pb.n_frags = kept[0];
    pb.n_bases = kept[1];
    if (pb.n_bases >= (1ull << 32)) return CFG_ERR_BAD_INPUT;
    const uint64_t words = (pb.n_bases + 31) / 32;
    if (!pb.ensure_packed(words + 4)) return CFG_ERR_OOM;
    if (cudaMemsetAsync(pb.packed, 0, 8 * (words + 4), s) != cudaSuccess) return CFG_ERR_CUDA;
    a.packed = pb.packed; a.frag_out = pb.frag_out;
    if (nc) k_parse_pack<<<pgrid, TPB, 0, s>>>(a);
    if (cudaGetLastError() != cudaSuccess) return CFG_ERR_CUDA;
    return CFG_OK;
}

}  // namespace cfg
