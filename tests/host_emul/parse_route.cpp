// parse_route.cpp -- the device text parser (csrc/cfg_parse.cu) run on a CPU by the words its
// passes leave for each other: a word per 16-byte group (pass A: the chunk's function before
// the group; pass C: the group's emissions) and one per 32 groups (bases and breaks of the
// chunk before them).  What is done with a group is the parser's own code
// (cfg_parse_thread.cuh); scans are loops.  Same exports as parse_emul/parse_emul.cpp.
#include "cfg_parse_thread.cuh"

#include <cstdlib>
#include <cstring>
#include <vector>

using namespace cfg::parse;

namespace {

Group group_at(const uint8_t* text, uint64_t bytes, uint64_t p) {
    Group g{};
    for (uint32_t i = 0; i < BPT; ++i)
        if (p + i < bytes) g.w[i / 4] |= (uint32_t)text[p + i] << (8 * (i % 4));
    return g;
}
uint32_t bytes_at(uint64_t bytes, uint64_t p) { return p >= bytes ? 0 : (uint32_t)umin64(BPT, bytes - p); }

struct HostOr64 {
    void operator()(uint64_t* w, uint64_t bits) const { *w |= bits; }
};

}  // namespace

extern "C" {

int parse_emul(const uint8_t* text, uint64_t bytes, int fastq, uint32_t k, uint64_t** words, uint64_t* n_bases,
               uint64_t** frag_off, uint32_t** frag_len, uint64_t* n_frags) {
    const FsmBits f = pack_fsm(fastq ? fastq_fsm() : fasta_fsm());
    const uint64_t nc = (bytes + CHUNK - 1) / CHUNK;
    std::vector<uint32_t> chunk_f(nc + 1), group_w(nc * TPB + 1), step_pre(nc * (TPB / 32) + 1);
    std::vector<unsigned long long> chunk_b(nc + 1), chunk_k(nc + 1);
    for (uint64_t c = 0; c < nc; ++c) {   // A
        Fn carry{0x03020100u, 4u};
        for (uint32_t t = 0; t < TPB; ++t) {
            const uint64_t p = c * CHUNK + (uint64_t)t * BPT;
            group_w[c * TPB + t] = fn_bits(carry);
            carry = fn_then(carry, thread_fn(f, group_at(text, bytes, p), bytes_at(bytes, p)));
        }
        chunk_f[c] = fn_bits(carry);
    }
    uint32_t st = f.start;                // B
    for (uint64_t c = 0; c < nc; ++c) { const uint32_t tf = chunk_f[c]; chunk_f[c] = st; st = f_at(tf, st); }
    for (uint64_t c = 0; c < nc; ++c) {   // C
        uint32_t carry = 0;
        for (uint32_t t = 0; t < TPB; ++t) {
            const uint64_t p = c * CHUNK + (uint64_t)t * BPT;
            if (t % 32 == 0) step_pre[(c * TPB + t) / 32] = carry;
            const Emits e = thread_emits(f, f_at(group_w[c * TPB + t], chunk_f[c]), group_at(text, bytes, p), bytes_at(bytes, p));
            group_w[c * TPB + t] = emits_word(e);
            carry += emits_counts(e);
        }
        chunk_b[c] = pre_bases(carry); chunk_k[c] = pre_breaks(carry);
    }
    unsigned long long rb = 0, rk = 0;    // D
    for (uint64_t c = 0; c < nc; ++c) {
        const unsigned long long x = chunk_b[c], y = chunk_k[c];
        chunk_b[c] = rb; chunk_k[c] = rk; rb += x; rk += y;
    }
    const uint64_t NB = rk;               // E
    std::vector<unsigned long long> brk_rank(NB + 1), frag_out(NB + 1);
    auto groups = [&](auto&& visit) {     // every group with the bases and breaks before it
        uint32_t pre = 0;
        for (uint64_t i = 0; i < nc * TPB; ++i) {
            if (i % 32 == 0) pre = step_pre[i / 32];
            const Emits e = word_emits(group_w[i]);
            visit(i, e, chunk_b[i / TPB] + pre_bases(pre), chunk_k[i / TPB] + pre_breaks(pre));
            pre += emits_counts(e);
        }
    };
    groups([&](uint64_t, Emits e, unsigned long long r, unsigned long long kk) { emit_breaks(e, r, kk, brk_rank.data()); });
    brk_rank[NB] = rb;
    std::vector<uint64_t> fo;             // F
    std::vector<uint32_t> fl;
    unsigned long long at = 0;
    for (uint64_t i = 0; i <= NB; ++i) {
        const unsigned long long L = brk_rank[i] - (i ? brk_rank[i - 1] : 0ull);
        frag_out[i] = L >= k + 1 ? at : ~0ull;
        if (L >= k + 1) { fo.push_back(at); fl.push_back((uint32_t)L); at += L; }
    }
    uint64_t* w = (uint64_t*)std::calloc((at + 31) / 32 + 4, 8);   // G
    uint64_t* o = (uint64_t*)std::malloc(8 * (fo.size() + 1));
    uint32_t* l = (uint32_t*)std::malloc(4 * (fl.size() + 1));
    if (!w || !o || !l) { std::free(w); std::free(o); std::free(l); return 1; }
    groups([&](uint64_t i, Emits e, unsigned long long r, unsigned long long kk) {
        emit_pack(e, group_at(text, bytes, i * BPT), r, kk, frag_out.data(), brk_rank.data(), w, HostOr64{});
    });
    if (!fo.empty()) { std::memcpy(o, fo.data(), 8 * fo.size()); std::memcpy(l, fl.data(), 4 * fl.size()); }
    *words = w; *n_bases = at; *frag_off = o; *frag_len = l; *n_frags = fo.size();
    return 0;
}

void parse_emul_free(void* p) { std::free(p); }

// runs_alike against the byte-by-byte meaning of it, on both machines with one table entry
// changed to every other value: runs of two and three bases and other bytes must move every
// state and emit as a run's first byte says.  -> entries it judged wrongly.
int runs_alike_mismatches() {
    int bad = 0;
    for (const Fsm& m0 : {fasta_fsm(), fastq_fsm()}) {
        for (uint32_t at = 0; at < m0.n * NCLASS * 2; ++at)
            for (uint32_t v = 0; v < 5; ++v) {
                Fsm m = m0;
                const uint32_t s = at / 2 / NCLASS, c = at / 2 % NCLASS;
                if (at & 1) { if (v > 2) continue; m.emit[s][c] = (uint8_t)v; } else m.next[s][c] = (uint8_t)v;
                bool alike = true;
                for (uint32_t st = 0; st < m.n; ++st)
                    for (uint32_t run = 0; run < 8; ++run) {   // three bytes, bit set: an other byte
                        const bool seq = m.emit[st][C_BASE] == E_BASE;
                        const uint32_t to = m.next[st][C_BASE];
                        uint32_t x = st;
                        for (uint32_t i = 0; i < 3; ++i) {
                            const uint32_t cl = run >> i & 1 ? C_OTHER : C_BASE;
                            alike = alike && m.emit[x][cl] == (!seq ? E_SKIP : cl == C_BASE ? E_BASE : E_BREAK);
                            x = m.next[x][cl];
                            alike = alike && x == to;
                        }
                    }
                bad += alike != runs_alike(m);
            }
    }
    return bad;
}

}  // extern "C"
