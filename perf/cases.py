"""The compaction path's work as programs use it: what is timed, and over which sizes.

Every case is one whole call sequence through the Python binding (the C ABI's entry
points): an input in one of the forms the library takes (packed bases in page-locked host
memory, FASTA or FASTQ text, packed bases in device memory), compacted to what the caller
keeps: the final maximal unitigs, or the lm-tigs with their discontinuity edges.  The
library leaves the order of its records open, so each pass also puts them in the order
of their sequences, which makes its output one definite array.

Inputs are synthetic, made from a seed on the GPU: genomes with repeated copies and
tandem repeats, and reads from both strands with substitutions, in the shapes of the
benchmark's workloads.
"""
import ctypes
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cuttlefish-private_b200", "python"))
import cfgpu  # noqa: E402

# path: how the input comes in and what is taken out
#   packed   host-packed fragments -> final unitigs          (cfg_submit_packed)
#   text     FASTA / FASTQ text -> final unitigs             (cfg_submit_text)
#   device   packed fragments in device memory -> unitigs    (cfg_submit_packed_device)
#   lmtigs   host-packed fragments -> lm-tigs and edges      (cfg_fetch: the reference's Subgraphs_Manager sinks)
#   batch    many genomes in one launch -> unitigs of each   (cfg_batch_*)
#   serve    a mix of jobs through the serving loop          (cfg_server_*)
#   noalloc  records of one small device-resident job        (cfg_partition_noalloc)


def _ref(name, path, bases, k, records, subgraphs=16384, l=20, repeats=False):
    return {"name": name, "path": path, "kind": "ref", "bases": bases, "records": records, "k": k, "l": l, "cutoff": 1,
            "subgraphs": subgraphs, "load": 100, "repeats": repeats}


def _reads(name, path, reads, lo, hi, coverage, k, subgraphs=16384, load=20):
    return {"name": name, "path": path, "kind": "reads", "reads": reads, "lo": lo, "hi": hi, "coverage": coverage, "k": k,
            "l": 20, "cutoff": 2, "subgraphs": subgraphs, "load": load}


def listed():
    return [
        # one small job partitioned on a caller's stream by a plugin that may not allocate
        _ref("noalloc_180k", "noalloc", 180_037, 31, 3),
        # a plasmid or a virus: the smallest jobs, where launches, copies and waits are the cost
        _ref("plasmid_50k", "packed", 50_021, 31, 1),
        # a small amplicon-sized FASTQ of quality-trimmed (ragged) reads
        _reads("fastq_trimmed_20k", "text", 20_011, 60, 150, 25, 27),
        # one bacterial genome: `build --ref -k 31 -c 1`, the benchmark's ref5m shape
        _ref("ref_5m", "packed", 4_999_983, 31, 1),
        # a fungal assembly from its FASTA file: wrapped lines, N runs, lowercase, a shorter k
        _ref("fasta_24m_k23", "text", 24_000_007, 23, 37, l=11),
        # lm-tigs and edges handed to the discontinuity-graph phases of a host program
        _ref("lmtigs_20m", "lmtigs", 20_000_033, 31, 5),
        # one lane of reads from its FASTQ file: `build --read -k 31 -c 2`
        _reads("fastq_2m", "text", 2_000_003, 150, 150, 30, 31, 32768, 15),
        # wide k-mers (four key words), as for nearly identical strains
        _ref("ref_12m_k127", "packed", 12_000_019, 127, 7, 16384),
        # a collection of genomes compacted together, the benchmark's batch shape
        {"name": "batch_40", "path": "batch", "kind": "ref", "jobs": 40, "lo": 500_000, "hi": 8_000_000, "k": 31, "l": 20,
         "cutoff": 1, "subgraphs": 16384, "tuned_subgraphs": 4096, "load": 100},
        # a server's queue: references and read sets of mixed size
        {"name": "serve_8", "path": "serve", "kind": "mix", "jobs": 8, "lo": 3_000_000, "hi": 6_000_000, "k": 31, "l": 20,
         "cutoff": 2, "subgraphs": 16384, "load": 20},
        # the benchmark's headline: 10 M reads at 30x, resident on the device
        _reads("reads_10m", "device", 10_000_000, 150, 150, 30, 31, 131072, 15),
        # a large repeat-rich reference at k = 63, the benchmark's ref500m shape
        _ref("ref_500m_k63", "packed", 500_000_003, 63, 20, 524288, repeats=True),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random())) | 1


def draw(rng):
    path = rng.choice(["noalloc", "packed", "packed", "packed", "text", "text", "device", "lmtigs", "batch", "serve"])
    if path == "batch":
        lo = _log(rng, 20_000, 1_000_000)
        return {"path": path, "kind": "ref", "jobs": rng.randint(3, 60), "lo": lo, "hi": lo * 8, "k": 31, "l": 20, "cutoff": 1,
                "subgraphs": 16384, "tuned_subgraphs": rng.choice([1024, 4096, 16384]), "load": 100}
    if path == "serve":
        lo = _log(rng, 50_000, 4_000_000)
        return {"path": path, "kind": "mix", "jobs": rng.randint(3, 9), "lo": lo, "hi": lo * 2, "k": 31, "l": 20, "cutoff": 2,
                "subgraphs": 16384, "load": 20}
    if path == "noalloc":
        return _drawn(_ref("", path, _log(rng, 4_000, 900_000), rng.choice([21, 31, 63, 127]), rng.randint(1, 9)))
    if path in ("packed", "text", "device") and rng.random() < 0.45:   # read sets
        k = rng.choice([21, 25, 27, 31, 31, 31, 47])
        n = _log(rng, 5_000, 4_000_000 if k < 32 else 500_000)
        lo, hi = rng.choice([(150, 150), (100, 100), (60, 150), (151, 251)])
        return _drawn(_reads("", path, n, lo, hi, rng.choice([12, 30, 60]), k, _subgraphs(n * hi, k), rng.choice([15, 20])))
    k = rng.choice([15, 23, 27, 31, 31, 31, 31, 41, 55, 63, 63, 95, 127])
    most = 2_000_000 if k == 15 else 60_000_000 if k < 31 else 200_000_000 if k <= 63 else 30_000_000
    bases = _log(rng, 20_000, min(most, 30_000_000) if path == "lmtigs" else most)
    c = _ref("", path, bases, k, min(rng.randint(1, 60), bases // 2000), 16384 if path == "lmtigs" else _subgraphs(bases, k),
             l=20 if k > 23 else 11 if k > 15 else 9, repeats=rng.random() < 0.4)
    return _drawn(c)


def _drawn(case):
    return {key: v for key, v in case.items() if key != "name"}


def _subgraphs(bases, k):
    """The subgraph count that cfgpu.tune_graph_count finds for such a job, roughly."""
    want = 16384
    while want < (524288 if k > 32 else 131072) and bases > want * (1000 if k > 32 else 11500):
        want *= 2
    return want


# ---------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1_000_003 + 17)
    return g


def _spans(g, n, count, lo, hi):
    """`count` disjoint spans of lo..hi bases in n: (starts, lengths, position in the span, span of each position)."""
    slot = n // max(1, count)
    lens = torch.randint(lo, hi + 1, (count,), generator=g, device="cuda").clamp_(max=max(1, slot - 1))
    starts = torch.arange(count, device="cuda") * slot + (torch.rand(count, generator=g, device="cuda", dtype=torch.float64) * (slot - lens)).long()
    owner = torch.repeat_interleave(torch.arange(count, device="cuda"), lens)
    first = torch.cumsum(lens, 0) - lens
    return starts, lens, torch.arange(owner.numel(), device="cuda") - first[owner], owner


def _substitute(g, codes, rate):
    hit = torch.rand(codes.shape, generator=g, device="cuda") < rate
    add = torch.randint(1, 4, codes.shape, generator=g, device="cuda", dtype=torch.uint8)
    return torch.where(hit, (codes + add) & 3, codes)


def _genome(g, n, repeats=False):
    """n base codes (0..3): random sequence with 1 % (repeats: 5 %) of it copies of other stretches at 1 % (5 %)
    substitutions, and with `repeats` 10 % tandem repeats of 2..50-base units."""
    x = torch.randint(0, 4, (n,), generator=g, device="cuda", dtype=torch.uint8)
    hi = max(60, min(5000, n // 20))
    lo = max(30, hi // 10)
    count = int(n * (0.05 if repeats else 0.01) / ((lo + hi) / 2)) + 1
    starts, lens, at, owner = _spans(g, n, count, lo, hi)
    src = (torch.rand(count, generator=g, device="cuda", dtype=torch.float64) * (n - hi)).long()
    x[starts[owner] + at] = _substitute(g, x[src[owner] + at], 0.05 if repeats else 0.01)
    if repeats:
        count = int(n * 0.1 / 5000) + 1
        starts, lens, at, owner = _spans(g, n, count, min(100, n // 40), min(10000, n // 8))
        unit = torch.randint(2, 51, (count,), generator=g, device="cuda")
        x[starts[owner] + at] = x[starts[owner] + at % unit[owner]]
    return x


def _cut(g, n, records):
    """Offsets of `records` records of unequal size in n bases."""
    w = torch.rand(records, generator=g, device="cuda", dtype=torch.float64) + 0.5
    off = torch.zeros(records + 1, dtype=torch.int64, device="cuda")
    off[1:] = (torch.cumsum(w, 0) / w.sum() * n).long()
    off[-1] = n
    return off


def _read_set(g, reads, lo, hi, coverage):
    """Codes of `reads` reads end to end, and their offsets: both strands, 0.5 % substitutions."""
    lens = torch.randint(lo, hi + 1, (reads,), generator=g, device="cuda")
    off = torch.zeros(reads + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(lens, 0)
    total = int(off[-1])
    genome = _genome(g, max(4 * hi, total // coverage))
    start = (torch.rand(reads, generator=g, device="cuda", dtype=torch.float64) * (genome.numel() - lens)).long()
    back = torch.randint(0, 2, (reads,), generator=g, device="cuda", dtype=torch.bool)
    out = torch.empty(total, dtype=torch.uint8, device="cuda")
    step = 1 << 20
    for r0 in range(0, reads, step):
        r1 = min(reads, r0 + step)
        a, b = int(off[r0]), int(off[r1])
        owner = torch.repeat_interleave(torch.arange(r0, r1, device="cuda"), lens[r0:r1])
        at = torch.arange(a, b, device="cuda") - off[owner]
        rev = back[owner]
        codes = genome[start[owner] + torch.where(rev, lens[owner] - 1 - at, at)]
        out[a:b] = _substitute(g, torch.where(rev, 3 - codes, codes), 0.005)
    return out, off


_ACGT = b"ACGT"


def _letters(codes):
    return torch.tensor(list(_ACGT), dtype=torch.uint8, device="cuda")[codes.int()]


def _pinned(t):
    h = torch.empty(t.numel(), dtype=torch.uint8, pin_memory=True)
    h.copy_(t.reshape(-1))
    return h


def _packed_input(codes, off, k):
    """cfg_pack_records on the records' letters, into page-locked memory."""
    text = _letters(codes).cpu()
    offs = off.cpu().numpy().astype(np.uint64)
    return cfgpu.PackedInput(None, k, pinned=True, data_offsets=(
        ctypes.cast(text.data_ptr(), ctypes.c_char_p), offs.ctypes.data_as(cfgpu.U64P), len(offs) - 1))


def _device_input(codes, off):
    """The packed layout in device memory: words with 4 words of padding, fragment offsets and lengths."""
    n = codes.numel()
    words = torch.zeros((n + 31) // 32 + 4, dtype=torch.int64, device="cuda")
    shifts = 62 - 2 * torch.arange(32, device="cuda")
    step = 1 << 28
    for a in range(0, n, step):
        part = codes[a:a + step]
        if part.numel() % 32:
            part = torch.nn.functional.pad(part, (0, 32 - part.numel() % 32))
        words[a // 32:a // 32 + part.numel() // 32] = (part.view(-1, 32).long() << shifts).sum(1)
    return words, n, off[:-1].contiguous(), (off[1:] - off[:-1]).to(torch.int32), off.numel() - 1


def _fasta(g, codes, off):
    """FASTA text of the records: lines of 70 bases, some N runs and lowercase stretches."""
    letters = _letters(codes)
    n = letters.numel()
    starts, lens, at, owner = _spans(g, n, n // 400_000 + 1, 1, min(200, n // 10))
    letters[starts[owner] + at] = ord("N")
    starts, lens, at, owner = _spans(g, n, n // 20_000 + 1, 20, min(2000, n // 10))
    letters[starts[owner] + at] |= 0x20
    parts = []
    for r in range(off.numel() - 1):
        s = letters[int(off[r]):int(off[r + 1])]
        head = torch.tensor(list(b">contig_%d\n" % r), dtype=torch.uint8, device="cuda")
        full = s.numel() // 70 * 70
        body = torch.nn.functional.pad(s[:full].view(-1, 70), (0, 1), value=10).reshape(-1)
        rest = torch.nn.functional.pad(s[full:], (0, 1), value=10) if full < s.numel() else s[:0]
        parts += [head, body, rest]
    return _pinned(torch.cat(parts))


def _fastq(g, codes, off):
    """FASTQ text of the reads: '@' and a nine-digit name, bases, '+', qualities."""
    reads = off.numel() - 1
    lens = off[1:] - off[:-1]
    size = 11 + 2 * (lens + 1) + 2                         # @ddddddddd\n  bases\n  +\n  qualities\n
    pos = torch.cumsum(size, 0) - size
    out = torch.empty(int(size.sum()), dtype=torch.uint8, device="cuda")
    out[pos] = ord("@")
    ids = torch.arange(reads, device="cuda")
    for d in range(9):
        out[pos + 1 + d] = (ids // 10 ** (8 - d) % 10 + ord("0")).to(torch.uint8)
    out[pos + 10] = 10
    out[pos + 11 + lens] = 10
    out[pos + 12 + lens] = ord("+")
    out[pos + 13 + lens] = 10
    out[pos + 14 + 2 * lens] = 10
    step = 1 << 20
    for r0 in range(0, reads, step):
        r1 = min(reads, r0 + step)
        a, b = int(off[r0]), int(off[r1])
        owner = torch.repeat_interleave(torch.arange(r0, r1, device="cuda"), lens[r0:r1])
        at = torch.arange(a, b, device="cuda") - off[owner] + pos[owner] + 11
        out[at] = _letters(codes[a:b])
        q = 73 - (torch.rand(b - a, generator=g, device="cuda") ** 4 * 38).to(torch.uint8)   # mostly I, down to #
        out[at + lens[owner] + 3] = q
    return _pinned(out)


def _job_sizes(case):
    """The jobs' bases: spread evenly over the logarithm of the range, large and small ones mixed."""
    n = case["jobs"]
    step = next(d for d in (7, 11, 13, 17) if n % d)
    return [int(case["lo"] * (case["hi"] / case["lo"]) ** ((i * step % n + 0.5) / n)) for i in range(n)]


def _unitig_bytes(case, bases):
    """Room for the unitigs of `bases` input bases, a line each: about the genome, and for read sets the variants that
    two reads share by chance and the breaks they make."""
    if case["kind"] == "ref":
        return int(bases * 1.25) + 65536
    depth = case["coverage"] / 30
    return int(bases / case["coverage"] * (1.6 + 0.6 * depth * depth * case["k"] / 31)) + 65536


def _lmtig_rows(case, bases):
    return int(bases * 2.8 / (case["k"] - case["l"] + 1)) + 4096   # about 2 / (k - l + 1) weak super k-mers a base


def _lmtig_room(case, bases):
    rows = _lmtig_rows(case, bases)
    return {"unitigs": _room(bases // 4 + 65536), "edges": torch.zeros((rows, 71), dtype=torch.uint8, device="cuda"),
            "labels": _room(bases + rows * case["k"] + 65536)}


def _room(n):
    """A caller's result buffer: device memory, or host memory when a small result is put in order there."""
    return torch.zeros(n, dtype=torch.uint8, device="cuda" if n > 1 << 18 else "cpu")


class _Program(dict):
    """What a program holds between calls; its context, batch or server is closed with it."""

    def __del__(self):
        for handle in ("server", "batch", "cx"):
            if handle in self:
                self[handle].close()


def prepare(case, seed):
    g = _gen(seed)
    path, k = case["path"], case["k"]
    s = _Program(case=case)
    if path == "batch":
        s["jobs"] = []
        for n in _job_sizes(case):
            x = _genome(g, n)
            s["jobs"].append(_packed_input(x, _cut(g, n, 1), k))
        s["room"] = _room(_unitig_bytes(case, sum(_job_sizes(case))))
        s["batch"] = cfgpu.Batch(k, case["l"], case["cutoff"], case["subgraphs"], table_load_pct=case["load"])
        s["batch"].set_tuning(local_div=8, cluster_threads=512, table_load_pct=case["load"], graph_count=case["tuned_subgraphs"])
    elif path == "serve":
        s["jobs"] = []
        for i, n in enumerate(_job_sizes(case)):
            if i % 2:   # a read set of n bases
                codes, off = _read_set(g, max(1, n // 150), 150, 150, 30)
                s["jobs"].append((_packed_input(codes, off, k), case["cutoff"], case["load"]))
            else:
                s["jobs"].append((_packed_input(_genome(g, n), _cut(g, n, 1), k), 1, 100))
        s["room"] = [_lmtig_room(case, n) for n in _job_sizes(case)]
        s["server"] = cfgpu.Server(slots=2, hbm_budget=24 << 30, batch_max_bases=16_000_000, small_job_bases=1_000_000)
    else:
        if case["kind"] == "reads":
            codes, off = _read_set(g, case["reads"], case["lo"], case["hi"], case["coverage"])
        else:
            codes = _genome(g, case["bases"], case["repeats"])
            off = _cut(g, case["bases"], case["records"])
        if path in ("packed", "lmtigs"):
            s["input"] = _packed_input(codes, off, k)
        elif path == "text":
            s["input"] = _fastq(g, codes, off) if case["kind"] == "reads" else _fasta(g, codes, off)
        else:
            s["input"] = _device_input(codes, off)
        if path == "noalloc":
            n, G = codes.numel(), case["subgraphs"]
            s["params"] = cfgpu.Params(k, case["l"], case["cutoff"], G, 0, 0, 0)
            s["records"] = torch.zeros(n, dtype=torch.int64, device="cuda")
            s["room"] = torch.zeros(n, dtype=torch.int64, device="cuda")
            s["bucket_off"] = torch.zeros(G + 1, dtype=torch.int32, device="cuda")
            s["n_records"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        else:
            bases = case["bases"] if case["kind"] == "ref" else case["reads"] * (case["lo"] + case["hi"]) // 2
            s["room"] = _lmtig_room(case, bases) if path == "lmtigs" else _room(_unitig_bytes(case, bases))
            s["cx"] = cfgpu.Compactor(k, case["l"], case["cutoff"], case["subgraphs"], table_load_pct=case["load"])
    return s


# ---------------------------------------------------------------------------- one pass

def _host(ptr, n):
    if not ptr or not n:
        return torch.empty(0, dtype=torch.uint8)
    return torch.frombuffer((ctypes.c_char * n).from_address(ptr), dtype=torch.uint8)


def _kmer_order(text, starts, k, group=None):
    """Order of the sequences at `starts` by (group, first k bases); a k-mer starts at most one sequence of a group."""
    order = None
    for a in range((k - 1) // 31 * 31, -1, -31):      # 31 bases per 64-bit key, the last ones first (stable sorts)
        m = min(31, k - a)
        c = text[(starts[:, None] + torch.arange(a, a + m, device="cuda"))].long()
        key = ((((c >> 1) ^ (c >> 2)) & 3) << (2 * torch.arange(m - 1, -1, -1, device="cuda"))).sum(1)
        order = torch.sort(key).indices if order is None else order[torch.sort(key[order], stable=True).indices]
    if group is not None:
        order = order[torch.sort(group[order], stable=True).indices]
    return order


def _put(room, rows):
    """The first rows of a result buffer, the rest cleared."""
    n = rows.shape[0]
    if n > room.shape[0]:
        raise RuntimeError("result buffer too small: %d of %d" % (room.shape[0], n))
    room[:n] = rows
    room[n:].zero_()
    return room


def _spread(text, starts, lens):
    """The spans text[starts : starts + lens], one after another."""
    first = torch.cumsum(lens, 0) - lens
    return text[torch.repeat_interleave(starts - first, lens) + torch.arange(int(lens.sum()), device="cuda")]


def _in_order(texts, k, room):
    """The sequences of FASTA texts (">0\\nSEQ\\n"), a line each, ordered by text and sequence."""
    if not room.is_cuda:
        lines = [sorted(x.numpy().tobytes().split(b"\n")[1::2]) for x in texts]
        return _put(room, torch.frombuffer(bytearray(b"".join(b + b"\n" for x in lines for b in x) or b"\0"), dtype=torch.uint8))
    text = torch.empty(sum(t.numel() for t in texts), dtype=torch.uint8, device="cuda")
    at, ends = 0, []
    for t in texts:
        text[at:at + t.numel()].copy_(t)
        at += t.numel()
        ends.append(at)
    nl = torch.nonzero(text == 10).squeeze(1)
    starts, lens = nl[0::2] + 1, nl[1::2] - nl[0::2]   # the newline included
    group = None
    if len(texts) > 1:
        group = torch.bucketize(starts, torch.tensor(ends, device="cuda"), right=True)
    order = _kmer_order(text, starts, k, group)
    return _put(room, _spread(text, starts[order], lens[order]))


def _lmtigs(r, k, room):
    """A fetched run's counts, trivial unitigs, and lm-tigs ordered by subgraph and label."""
    c = r.counts
    out = {"counts": np.array([c.n_bases, c.n_records, c.n_instances, c.n_vertices, c.n_isolated, c.n_phantom, c.n_trivial, c.n_icc,
                               c.n_lmtig, c.fasta_bytes, c.lmtig_bytes], dtype=np.int64),
           "unitigs": _in_order([_host(r.fasta, c.fasta_bytes)], k, room["unitigs"])}
    size = ctypes.sizeof(cfgpu.Lmtig)
    rec = _host(ctypes.cast(r.lmtigs, ctypes.c_void_p).value, c.n_lmtig * size).cuda().view(-1, size)
    text = _host(r.lmtig_text, c.lmtig_bytes).cuda()
    off = rec[:, 64:72].contiguous().view(torch.int64).squeeze(1)
    lens = rec[:, 72:76].contiguous().view(torch.int32).squeeze(1).long()
    g = rec[:, 76].long() | (rec[:, 77].long() << 8)
    order = _kmer_order(text, off, k, g)
    out["edges"] = _put(room["edges"], torch.cat([rec[:, :64], rec[:, 72:79]], 1)[order])     # u, v, length, subgraph, flags
    out["labels"] = _put(room["labels"], _spread(text, off[order], lens[order]))
    return out


def run(state):
    case = state["case"]
    path, k = case["path"], case["k"]
    if path == "noalloc":
        words, n, off, lens, frags = state["input"]
        stream = torch.cuda.current_stream().cuda_stream
        rc = cfgpu.load().cfg_partition_noalloc(
            torch.cuda.current_device(), ctypes.byref(state["params"]), words.data_ptr(), n, off.data_ptr(), lens.data_ptr(), frags,
            state["records"].data_ptr(), n, state["bucket_off"].data_ptr(), state["n_records"].data_ptr(), stream)
        if rc:
            raise RuntimeError("cfg_partition_noalloc: %d" % rc)
        count = int(state["n_records"])
        return {"records": _put(state["room"], torch.sort(state["records"][:count]).values), "bucket_off": state["bucket_off"], "n": count}
    if path == "batch":
        b = state["batch"]
        b.submit(state["jobs"])
        b.run()
        b.unitigs()
        texts, units = [], []
        for j in range(len(state["jobs"])):
            ptr, n, u = b.job_unitigs_raw(j)
            texts.append(_host(ptr, n).cuda())
            units.append(u)
        return {"unitigs": _in_order(texts, k, state["room"]), "n": np.array(units, dtype=np.int64)}
    if path == "serve":
        sv = state["server"]
        tickets = [sv.submit(p, k, case["l"], cutoff, case["subgraphs"], load) for p, cutoff, load in state["jobs"]]
        out = {}
        for _ in tickets:
            t, r, _tm = sv.wait_any_raw()
            j = tickets.index(t)
            out["job%d" % j] = _lmtigs(r, k, state["room"][j])
            sv.release(t)
        return out
    cx = state["cx"]
    if path == "text":
        cx.submit_text_ptr(state["input"].data_ptr(), state["input"].numel())
    elif path == "device":
        words, n, off, lens, frags = state["input"]
        cx.submit_device(words.data_ptr(), n, off.data_ptr(), lens.data_ptr(), frags)
    else:
        cx.submit(state["input"])
    cx.run()
    if path == "lmtigs":
        return _lmtigs(cx.fetch_raw(), k, state["room"])
    ptr, n, units, _ms = cx.unitigs_raw()
    return {"unitigs": _in_order([_host(ptr, n)], k, state["room"]), "n": units}


def work(case):
    """The input read once (2 bits a base packed, or the text) and the outputs written once (about a byte per distinct
    base: the genome; records of 8 bytes about every 6 bases for noalloc, lm-tigs of 88 bytes with their label)."""
    k, path = case["k"], case["path"]
    if path in ("batch", "serve"):
        n = sum(_job_sizes(case))
        return {"bytes": n / 4 + (n if path == "batch" else n * 0.5 * (1 + (88 + k) / 6)), "flops": 0}
    if case["kind"] == "reads":
        n = case["reads"] * (case["lo"] + case["hi"]) / 2
        genome, text = n / case["coverage"], 2 * n + 15 * case["reads"]
    else:
        n = genome = case["bases"]
        text = n * 71 / 70
    out = {"noalloc": 8 * n / 6, "lmtigs": n + (88 + k) * n / 6}.get(path, genome)
    return {"bytes": (text if path == "text" else n / 4) + out, "flops": 0}
