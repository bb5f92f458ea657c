// cfg_parse_thread.cuh -- what one thread of the device text parser (cfg_parse.cu) does
// with its 16 bytes, as __host__ __device__ code: the kernels run these steps on the
// GPU, and host harnesses in the tests run them over every group of a text on a CPU.  The
// steps are thread_fn, thread_emits, emits_word and its inverse, emit_breaks and emit_pack;
// thread_transfer, thread_counts, thread_breaks, thread_pack and thread_span put them
// together for the harness that checks one step at a time, and no kernel calls those.
//
// Bytes have five classes (newline, '>', a base letter, '\r', other); a finite-state
// machine over the classes (the line structure of FASTA or FASTQ) gives each byte an
// emission: skipped, a base, or a break (a non-ACGT character, a record boundary).
//
// A group is never walked byte by byte.  In both machines (runs_alike, checked when they are
// compiled) a run of base and other bytes
// moves every state once (one class map, idempotent) and emits alike from its first byte to
// its last -- bases and breaks from the states of a sequence line, nothing from the others
// -- so only the delimiters ('\n', '\r', and '>' where it is one) step the state.  Word-wise
// byte compares (SWAR) find them and the base letters as 16-bit masks; the group's emissions
// are two such masks, and its 2-bit codes are cut out of all 16 bytes' codes by runs.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CFG_PHD __host__ __device__ __forceinline__
#else
#define CFG_PHD inline
#endif

namespace cfg {
namespace parse {

constexpr uint32_t CHUNK = 4096, TPB = 256, BPT = CHUNK / TPB;   // bytes per thread: 16
enum : uint32_t { C_NL = 0, C_GT = 1, C_BASE = 2, C_CR = 3, C_OTHER = 4, NCLASS = 5 };
enum : uint32_t { E_SKIP = 0, E_BASE = 1, E_BREAK = 2 };

CFG_PHD uint32_t byte_perm(uint32_t x, uint32_t y, uint32_t s) {   // bytes of {y, x} picked by s's four nibbles
#ifdef __CUDA_ARCH__
    return __byte_perm(x, y, s);
#else
    const uint64_t v = ((uint64_t)y << 32) | x;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= (uint32_t)(v >> (8 * ((s >> (4 * i)) & 7)) & 0xFF) << (8 * i);
    return r;
#endif
}
// A transfer function of at most 5 states as bytes: state s's image in byte s of lo, state
// 4's in the low byte of hi (the rest of hi is unspecified).
struct Fn { uint32_t lo, hi; };
CFG_PHD Fn fn_of(uint32_t f) {   // from 3 bits per state
    return Fn{(f & 7u) | ((f << 5) & 0x700u) | ((f << 10) & 0x70000u) | ((f << 15) & 0x7000000u), (f >> 12) & 7u};
}
CFG_PHD uint32_t fn_bits(Fn f) {   // to 3 bits per state
    return (f.lo & 7u) | ((f.lo >> 5) & 0x38u) | ((f.lo >> 10) & 0x1C0u) | ((f.lo >> 15) & 0xE00u) | ((f.hi & 7u) << 12);
}
// first f, then g: f's images, as nibbles, are the byte selectors into g
CFG_PHD Fn fn_then(Fn f, Fn g) {
    const uint32_t y = f.lo | (f.lo >> 4);
    return Fn{byte_perm(g.lo, g.hi, byte_perm(y, 0, 0x4420u)), byte_perm(g.lo, g.hi, f.hi & 7u)};
}

// The tables of an FSM of at most 5 states packed into registers: entry (class c, state s)
// at index i = 5 c + s, its next state in 3 bits (bits 3i.. of nx_lo for i < 21, of nx_hi
// above) and its emission in 2 bits of em.  A lookup is a few shifts on values every
// thread holds, where an indexed table (in the kernel's parameters or in memory) would
// serialise the warp's lanes over their distinct (state, class) pairs.
struct FsmBits {
    unsigned long long nx_lo, nx_hi, em;
    // class c's whole next-state map as a transfer function (3 bits per state): bits 15c..
    // of cf_lo for c < 4, cf_hi for c = 4
    unsigned long long cf_lo;
    uint32_t cf_hi;
    uint32_t n, start;
    // word-wise groups: gt_other -- '>' has the next states and emissions of an other byte in
    // every state (it is then no delimiter); seq_mask bit s -- runs that start in state s emit
    // (base: E_BASE, other: E_BREAK; from the other states E_SKIP).  Of the machine, read by no
    // step: loop_mask bit s -- state s stays s on a base and on an other byte; bo_idem -- bases
    // and other bytes have one class map, and it is idempotent
    uint32_t loop_mask, gt_other, bo_idem, seq_mask;
    Fn run, nl, cr, gt;   // the class maps of a run, '\n', '\r' and '>'
};

CFG_PHD uint32_t fsm_next(const FsmBits& f, uint32_t st, uint32_t cl) {
    const uint32_t i = 5 * cl + st;
    return i < 21 ? (uint32_t)(f.nx_lo >> (3 * i)) & 7u : (uint32_t)(f.nx_hi >> (3 * (i - 21))) & 7u;
}
CFG_PHD uint32_t fsm_emit(const FsmBits& f, uint32_t st, uint32_t cl) {
    return (uint32_t)(f.em >> (2 * (5 * cl + st))) & 3u;
}
CFG_PHD uint32_t class_fn(const FsmBits& f, uint32_t cl) {
    return cl < 4 ? (uint32_t)(f.cf_lo >> (15 * cl)) & 0x7FFFu : f.cf_hi;
}
CFG_PHD uint32_t byte_class(uint32_t c) {
    if (c == '\n') return C_NL;
    if (c == '>') return C_GT;
    if (c == '\r') return C_CR;
    const uint32_t u = c & 0xDF;
    return (u == 'A' || u == 'C' || u == 'G' || u == 'T') ? C_BASE : C_OTHER;
}
CFG_PHD uint32_t base_code(uint32_t c) {   // A0 C1 G2 T3 (case-insensitive)
    const uint32_t u = c & 0xDF;
    return u == 'A' ? 0 : u == 'C' ? 1 : u == 'G' ? 2 : 3;
}
CFG_PHD uint32_t f_at(uint32_t f, uint32_t s) { return (f >> (3 * s)) & 7; }
CFG_PHD uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }
// first f, then g
CFG_PHD uint32_t compose(uint32_t f, uint32_t g, uint32_t n) {
    uint32_t h = 0;
    for (uint32_t s = 0; s < n; ++s) h |= f_at(g, f_at(f, s)) << (3 * s);
    return h;
}
CFG_PHD uint32_t identity(uint32_t n) {
    uint32_t h = 0;
    for (uint32_t s = 0; s < n; ++s) h |= s << (3 * s);
    return h;
}

CFG_PHD uint32_t popc32(uint32_t x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__popc(x);
#else
    return (uint32_t)__builtin_popcount(x);
#endif
}

// A thread's 16 bytes as four little-endian words: byte i is bits 8(i%4).. of w[i/4].
struct Group { uint32_t w[4]; };

CFG_PHD uint32_t byte_at(const Group& g, uint32_t i) { return (g.w[i >> 2] >> (8 * (i & 3))) & 0xFFu; }

// 0x80 in every byte of x that equals the byte value b, 0 in every other byte (exact:
// no byte's sum carries into the next)
CFG_PHD uint32_t eq_bytes(uint32_t x, uint32_t b) {
    const uint32_t y = x ^ (b * 0x01010101u);
    return ~(((y & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | y) & 0x80808080u;
}

// The top bits of x's four bytes as bits 0..3.
CFG_PHD uint32_t top_bits(uint32_t x) { return ((x & 0x80808080u) * 0x00204081u) >> 28; }

// Whether the group may hold a delimiter: some byte below 0x0E ('\n' and '\r' are) or,
// unless it acts as an other byte, a '>'.
CFG_PHD bool maybe_delimiter(const FsmBits& f, const Group& g) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m |= (g.w[i] - 0x0E0E0E0Eu) & ~g.w[i];
        if (!f.gt_other) {
            const uint32_t y = g.w[i] ^ 0x3E3E3E3Eu;
            m |= (y - 0x01010101u) & ~y;
        }
    }
    return (m & 0x80808080u) != 0;
}
// Bit i: byte i equals b.
CFG_PHD uint32_t eq_mask(const Group& g, uint32_t b) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) m |= top_bits(eq_bytes(g.w[i], b)) << (4 * i);
    return m;
}
// The delimiters among the group's first nb bytes, by kind.
struct Delims { uint32_t nl, cr, gt; };
CFG_PHD Delims delims(const FsmBits& f, const Group& g, uint32_t nb) {
    const uint32_t v = nb >= BPT ? 0xFFFFu : (1u << nb) - 1u;
    return Delims{eq_mask(g, '\n') & v, eq_mask(g, '\r') & v, f.gt_other ? 0u : eq_mask(g, '>') & v};
}
// Each byte's 2-bit code ((c >> 1) ^ (c >> 2)) & 3: a base letter's (A 0x41, C 0x43, G 0x47,
// T 0x54 and their lower-case forms: A0 C1 G2 T3), any value for other bytes.
CFG_PHD uint32_t codes4(uint32_t w) { return ((w >> 1) ^ (w >> 2)) & 0x03030303u; }
// Bit i: byte i is a base letter -- the letter of its code, either case.
CFG_PHD uint32_t acgt_mask(const Group& g) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t c = codes4(g.w[i]), y = c | (c >> 4);
        const uint32_t letter = byte_perm(0x54474341u, 0, byte_perm(y, 0, 0x4420u));
        const uint32_t d = (g.w[i] ^ letter) & 0xDFDFDFDFu;
        m |= top_bits(~(((d & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | d)) << (4 * i);
    }
    return m;
}

CFG_PHD uint32_t low_bit(uint32_t x) {   // index of the lowest set bit (x != 0)
#ifdef __CUDA_ARCH__
    return (uint32_t)__ffs((int)x) - 1u;
#else
    return (uint32_t)__builtin_ctz(x);
#endif
}

// The transfer function of nb bytes (nb <= 16): the runs' map and the delimiters', in order.
CFG_PHD Fn thread_fn(const FsmBits& f, const Group& g, uint32_t nb) {
    if (nb == BPT && !maybe_delimiter(f, g)) return f.run;
    const Delims d = delims(f, g, nb);
    Fn fn = Fn{0x03020100u, 4u};
    uint32_t pos = 0;
    for (uint32_t m = d.nl | d.cr | d.gt; m; m &= m - 1) {
        const uint32_t p = low_bit(m), b = m & (0u - m);
        if (p > pos) fn = fn_then(fn, f.run);
        fn = fn_then(fn, d.nl & b ? f.nl : d.cr & b ? f.cr : f.gt);
        pos = p + 1;
    }
    if (nb > pos) fn = fn_then(fn, f.run);
    return fn;
}
CFG_PHD uint32_t thread_transfer(const FsmBits& f, const Group& g, uint32_t nb) { return fn_bits(thread_fn(f, g, nb)); }

// Bases (low 16 bits) and breaks (high 16 bits) within one chunk, of at most 4096 bytes.
CFG_PHD uint32_t pre_pack(uint32_t eb, uint32_t ek) { return eb | (ek << 16); }
CFG_PHD uint32_t pre_bases(uint32_t p) { return p & 0xFFFFu; }
CFG_PHD uint32_t pre_breaks(uint32_t p) { return p >> 16; }

// What the group's nbytes bytes emit from state st: bit i of base (brk) -- byte i is a base
// (a break).
struct Emits { uint32_t base, brk; };
CFG_PHD Emits thread_emits(const FsmBits& f, uint32_t st, const Group& g, uint32_t nbytes) {
    if (nbytes == BPT && !maybe_delimiter(f, g)) {
        if (!((f.seq_mask >> st) & 1)) return Emits{0u, 0u};
        const uint32_t a = acgt_mask(g);
        return Emits{a, a ^ 0xFFFFu};
    }
    const Delims d = delims(f, g, nbytes);
    uint32_t seq = 0, brk = 0, pos = 0;   // bytes of emitting runs; breaking delimiters
    for (uint32_t m = d.nl | d.cr | d.gt; m; m &= m - 1) {
        const uint32_t p = low_bit(m), b = m & (0u - m);
        if (p > pos) {
            if ((f.seq_mask >> st) & 1) seq |= b - (1u << pos);
            st = f_at(class_fn(f, C_BASE), st);
        }
        const uint32_t cl = d.nl & b ? (uint32_t)C_NL : d.cr & b ? (uint32_t)C_CR : (uint32_t)C_GT;
        if (fsm_emit(f, st, cl) == E_BREAK) brk |= b;
        st = fsm_next(f, st, cl);
        pos = p + 1;
    }
    if (nbytes > pos && ((f.seq_mask >> st) & 1)) seq |= (1u << nbytes) - (1u << pos);
    if (!seq) return Emits{0u, brk};
    const uint32_t a = acgt_mask(g);
    return Emits{a & seq, brk | (seq & ~a)};
}

// A group's emissions as one word: what pass C leaves for E and G.
CFG_PHD uint32_t emits_word(Emits e) { return e.base | (e.brk << 16); }
CFG_PHD Emits word_emits(uint32_t m) { return Emits{m & 0xFFFFu, m >> 16}; }
// Its bases and breaks.
CFG_PHD uint32_t emits_counts(Emits e) { return pre_pack(popc32(e.base), popc32(e.brk)); }

// Bases and breaks the group emits from state st.
CFG_PHD void thread_counts(const FsmBits& f, uint32_t st, const Group& g, uint32_t nbytes, uint32_t& nb, uint32_t& nk) {
    const Emits e = thread_emits(f, st, g, nbytes);
    nb = popc32(e.base); nk = popc32(e.brk);
}

// The rank (bases before it) of each break the group emits: r bases and kk breaks precede
// the group's first byte.
CFG_PHD void emit_breaks(Emits e, unsigned long long r, unsigned long long kk, unsigned long long* brk_rank) {
    for (uint32_t m = e.brk; m; m &= m - 1) brk_rank[kk++] = r + popc32(e.base & ((m & (0u - m)) - 1u));
}
CFG_PHD void thread_breaks(const FsmBits& f, uint32_t st, const Group& g, uint32_t nbytes, unsigned long long r,
                           unsigned long long kk, unsigned long long* brk_rank) {
    emit_breaks(thread_emits(f, st, g, nbytes), r, kk, brk_rank);
}

// 2-bit codes of the group's 16 bytes, byte 0's in bits 31:30.
CFG_PHD uint32_t pack16(const Group& g) {
    uint32_t p = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) p = (p << 8) | ((codes4(g.w[i]) * 0x40100401u) >> 24);
    return p;
}

// Where the packed stream wants base i of fragment kk: out[kk] + (bases before it in the
// fragment); ~0 for a dropped fragment.
struct FragPos {
    unsigned long long out, first;   // the fragment's output start, the rank of its first base
};
CFG_PHD FragPos frag_pos(const unsigned long long* frag_out, const unsigned long long* brk_rank, unsigned long long kk) {
    return FragPos{frag_out[kk], kk ? brk_rank[kk - 1] : 0ull};
}

// The group's bases into the packed stream (MSB-first, 32 per word, every word zero
// before the pass): r bases and kk breaks precede the group.  or64(word pointer, bits)
// merges bits into a word (an atomic on the GPU: a word's bases may come from two threads).
// Each stretch of bases between two breaks is one fragment's: its runs of adjacent bytes
// are cut out of the 16 codes, joined, and merged into at most two words.
template <class Or64>
CFG_PHD void emit_pack(Emits e, const Group& g, unsigned long long r, unsigned long long kk,
                       const unsigned long long* frag_out, const unsigned long long* brk_rank, uint64_t* packed, Or64 or64) {
    const uint64_t codes = (uint64_t)pack16(g) << 32;   // byte 0's at bits 63:62
    uint32_t brk = e.brk;
    for (uint32_t left = e.base; left;) {
        const uint32_t b = brk & (0u - brk);                         // the next break, 0: none
        uint32_t part = b ? left & (b - 1u) : left;                  // bases before it
        left ^= part;
        brk ^= b;
        if (part) {
            const FragPos fp = frag_pos(frag_out, brk_rank, kk);
            const uint32_t total = popc32(part);
            if (fp.out != ~0ull) {
                uint64_t acc = 0;
                uint32_t n = 0;
                while (part) {
                    const uint32_t lo = low_bit(part), len = low_bit(~(part >> lo));
                    acc |= ((codes << (2 * lo)) & ~(~0ull >> (2 * len))) >> (2 * n);   // len <= 16
                    n += len;
                    part &= ~(((1u << len) - 1u) << lo);
                }
                const unsigned long long q = fp.out + (r - fp.first);
                const uint32_t o = (uint32_t)(q & 31);
                or64(packed + (q >> 5), acc >> (2 * o));
                if (o + n > 32) or64(packed + (q >> 5) + 1, acc << (64 - 2 * o));
            }
            r += total;
        }
        ++kk;
    }
}
template <class Or64>
CFG_PHD void thread_pack(const FsmBits& f, uint32_t st, const Group& g, uint32_t nbytes, unsigned long long r,
                         unsigned long long kk, uint32_t nb, uint32_t nk, const unsigned long long* frag_out,
                         const unsigned long long* brk_rank, uint64_t* packed, Or64 or64) {
    (void)nk;
    if (nb) emit_pack(thread_emits(f, st, g, nbytes), g, r, kk, frag_out, brk_rank, packed, or64);
}

// After pass D: bases and breaks before thread t's bytes (r, kk) and its own (nb, nk),
// from pass C's per-thread prefixes (the next thread's, or the chunk's totals for the
// last thread of a chunk); chunk_b / chunk_k hold the chunks' exclusive prefixes, with
// the totals at index n_chunks.
struct ThreadSpan { unsigned long long r, kk; uint32_t nb, nk; };
CFG_PHD ThreadSpan thread_span(const uint32_t* thread_pre, const unsigned long long* chunk_b,
                               const unsigned long long* chunk_k, uint64_t c, uint32_t t) {
    const uint64_t i = c * TPB + t;
    const uint32_t p = thread_pre[i];
    const unsigned long long cb = chunk_b[c], ck = chunk_k[c];
    uint32_t eb1, ek1;
    if (t + 1 < TPB) {
        const uint32_t q = thread_pre[i + 1];
        eb1 = pre_bases(q); ek1 = pre_breaks(q);
    } else {
        eb1 = (uint32_t)(chunk_b[c + 1] - cb); ek1 = (uint32_t)(chunk_k[c + 1] - ck);
    }
    return ThreadSpan{cb + pre_bases(p), ck + pre_breaks(p), eb1 - pre_bases(p), ek1 - pre_breaks(p)};
}

// ---------------------------------------------------------------------------------------
// The machines (host): their tables, and the packed form the kernels read.

// Up to 8 states; a transfer function packs the image of each state in 3 bits.
struct Fsm {
    uint8_t next[8][NCLASS];
    uint8_t emit[8][NCLASS];
    uint32_t n, start;
};

// What the word-wise steps take for granted: bases and other bytes have one class map, and it
// is idempotent; a run of them emits its bases and breaks on its other bytes, or nothing, and
// does the same from its second byte on as from its first.
constexpr bool runs_alike(const Fsm& m) {
    for (uint32_t st = 0; st < m.n; ++st) {
        const uint32_t nx = m.next[st][C_BASE];
        if (m.next[st][C_OTHER] != nx || m.next[nx][C_BASE] != nx) return false;
        const bool seq = m.emit[st][C_BASE] == E_BASE;
        if (m.emit[st][C_BASE] != (seq ? E_BASE : E_SKIP) || m.emit[st][C_OTHER] != (seq ? E_BREAK : E_SKIP)) return false;
        if ((m.emit[nx][C_BASE] == E_BASE) != seq) return false;
    }
    return true;
}

inline FsmBits pack_fsm(const Fsm& m) {
    FsmBits b{};
    b.n = m.n; b.start = m.start;
    for (uint32_t c = 0; c < NCLASS; ++c) {
        uint32_t F = 0;
        for (uint32_t st = 0; st < m.n; ++st) {
            const uint32_t i = 5 * c + st;
            if (i < 21) b.nx_lo |= (unsigned long long)m.next[st][c] << (3 * i);
            else b.nx_hi |= (unsigned long long)m.next[st][c] << (3 * (i - 21));
            b.em |= (unsigned long long)m.emit[st][c] << (2 * i);
            F |= (uint32_t)m.next[st][c] << (3 * st);
        }
        if (c < 4) b.cf_lo |= (unsigned long long)F << (15 * c); else b.cf_hi = F;
    }
    b.gt_other = 1;
    b.bo_idem = 1;
    for (uint32_t st = 0; st < m.n; ++st) {
        if (m.next[st][C_BASE] == st && m.next[st][C_OTHER] == st) b.loop_mask |= 1u << st;
        if (m.next[st][C_GT] != m.next[st][C_OTHER] || m.emit[st][C_GT] != m.emit[st][C_OTHER]) b.gt_other = 0;
        if (m.next[st][C_BASE] != m.next[st][C_OTHER] || m.next[m.next[st][C_BASE]][C_BASE] != m.next[st][C_BASE])
            b.bo_idem = 0;
        if (m.emit[st][C_BASE] == E_BASE) b.seq_mask |= 1u << st;
    }
    b.run = fn_of(class_fn(b, C_BASE)); b.nl = fn_of(class_fn(b, C_NL));
    b.cr = fn_of(class_fn(b, C_CR)); b.gt = fn_of(class_fn(b, C_GT));
    return b;
}

constexpr Fsm fasta_fsm() {
    // states: 0 line start before any record, 1 inside such a line, 2 header,
    // 3 line start inside a record, 4 sequence line
    Fsm m{};
    m.n = 5; m.start = 0;
    auto set = [&](uint32_t s, uint32_t c, uint32_t nx, uint32_t e) { m.next[s][c] = (uint8_t)nx; m.emit[s][c] = (uint8_t)e; };
    for (uint32_t c = 0; c < NCLASS; ++c) {
        set(0, c, 1, E_SKIP); set(1, c, 1, E_SKIP); set(2, c, 2, E_SKIP);
        set(3, c, 4, E_BREAK); set(4, c, 4, E_BREAK);
    }
    set(0, C_NL, 0, E_SKIP); set(0, C_CR, 0, E_SKIP); set(0, C_GT, 2, E_BREAK);
    set(1, C_NL, 0, E_SKIP);
    set(2, C_NL, 3, E_SKIP);
    set(3, C_NL, 3, E_SKIP); set(3, C_GT, 2, E_BREAK); set(3, C_BASE, 4, E_BASE);
    set(4, C_NL, 3, E_SKIP); set(4, C_BASE, 4, E_BASE);
    return m;
}

constexpr Fsm fastq_fsm() {
    // states: 0 before a record (blank lines skipped), 1 header line, 2 sequence line,
    // 3 '+' line, 4 quality line
    Fsm m{};
    m.n = 5; m.start = 0;
    auto set = [&](uint32_t s, uint32_t c, uint32_t nx, uint32_t e) { m.next[s][c] = (uint8_t)nx; m.emit[s][c] = (uint8_t)e; };
    for (uint32_t c = 0; c < NCLASS; ++c) {
        set(0, c, 1, E_SKIP); set(1, c, 1, E_SKIP); set(2, c, 2, E_BREAK); set(3, c, 3, E_SKIP); set(4, c, 4, E_SKIP);
    }
    set(0, C_NL, 0, E_SKIP); set(0, C_CR, 0, E_SKIP);
    set(1, C_NL, 2, E_SKIP);
    set(2, C_NL, 3, E_BREAK); set(2, C_BASE, 2, E_BASE);
    set(3, C_NL, 4, E_SKIP);
    set(4, C_NL, 0, E_SKIP);
    return m;
}

static_assert(runs_alike(fasta_fsm()) && runs_alike(fastq_fsm()), "the word-wise steps read both machines' runs alike");

}  // namespace parse
}  // namespace cfg
