"""Paths of the compaction that ordinary inputs of a test's size do not take, each forced by an input made for it and
compared with the oracle, the host packer or a plain run: the line between every two table shapes, labels past a warp's
copy, a record buffer and an output arena that prove too small, text past a gigabyte, the widest table of a batch."""
import numpy as np
import pytest

import cfgpu
import orc
import synth
from test_gpu_batch import check_batch
from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def instances(rng, n, k, l):
    """Two fragments with n k-mer instances in one subgraph: runs are cut every k - l positions, and a cut's k-mer counts
    on both sides of it."""
    m = max(x for x in range(n) if x + x // (k - l) <= n - 2)
    return [synth.random_seq(rng, x + k - 1) for x in (m, n - m - m // (k - l))]


@pytest.mark.parametrize("k,n", [(31, n) for n in (2047, 2048, 2049, 2520, 2521, 2522, 5040, 5041, 5042, 16383, 16384, 16385)] +
                         [(63, n) for n in (4799, 4800, 4801)] + [(127, n) for n in (3209, 3210, 3211)])
def test_table_shape_lines(k, n):
    """One subgraph of n k-mer instances to either side of a line: for k <= 31 where tables begin to fill to 0.62 (2048
    instances), the last of 4096 slots (2521) and of 8192 (5041, then a cluster), the last cluster (16384, then the
    arena); beyond, the last one-CTA table.  The count is a bound at the default load, so no table overflows."""
    counts = compare(instances(np.random.default_rng(600 + n), n, k, 20), k, 20, 1, 1)
    assert counts.n_instances == n and counts.n_retries == 0


@pytest.mark.parametrize("flip", [False, True])
def test_long_lmtig_labels(flip):
    """Two subgraphs at k = 127 leave lm-tigs of up to 770 bases, of which the collation writes pieces past 256 bases a
    warp at a time, forwards and reversed, inside a chain and at its tail."""
    k = 127
    g = synth.genome_with_repeats(np.random.default_rng(80), 200_000, n_copies=20, n_pal=10)
    recs = [synth.rc(g) if flip else g]
    o = orc.OracleRun(recs, k, 20, 1, 2)
    assert sum(n for (_, label, *_), n in o.lmtigs.items() if len(label) > 256 + k) > 50
    packed = cfgpu.PackedInput(recs, k)
    with cfgpu.Compactor(k, 20, 1, 2) as cx:
        cx.submit(packed)
        cx.run()
        fa, _ = cx.unitigs()
    packed.close()
    assert orc.fasta_multiset(fa) == orc.OracleRun(recs, k, 20, 1, 1).fasta_records()


def test_record_buffer_overflow():
    """k = 23, l = 20 makes half a record a base, twice what the record buffer is sized for: the sort and the plan queued
    behind the partition find nothing to do, and the run starts over with a larger buffer."""
    counts = compare([synth.random_seq(np.random.default_rng(81), 560_000)], 23, 20, 1, 16384)
    assert counts.n_records > max(560_000 // 4 + 1024, (1 << 21) // 8)   # the buffer's first size, whole 2 MiB


@pytest.mark.parametrize("G,candidates,keep", [(8, 150_000, 12_000), (1024, 400_000, 4_000)])
def test_output_arena_overflow(G, candidates, keep):
    """Fragments of one record, all of which fall to one output stripe: its slice of the FASTA arena is too small, and
    the plan and every table are made again over larger arenas."""
    k, stripes = 31, min(32, G)
    rng = np.random.default_rng(82)
    frags = [synth.random_seq(rng, k + 1) for _ in range(candidates)]
    off = (np.arange(candidates + 1) * (k + 1)).astype(np.uint64)
    data = "".join(frags).encode()
    o = orc.OracleArrays(data, off.ctypes.data_as(cfgpu.U64P), candidates, k, 20, 1, G)
    out = np.ones(candidates, dtype=bool)
    np.logical_and.at(out, (o.records["src"] // (k + 1)).astype(np.int64), o.records["g"] % stripes == 0)
    recs = [frags[i] for i in np.flatnonzero(out)]
    assert len(recs) > keep
    # the run's first estimate of one stripe's share of the FASTA, with every allowance for growth
    need = len(recs) * (k + 1) + (3 * len(recs) + 1024) * 8 + (1 << 20)
    assert len(recs) * (k + 5) > (need // stripes * 9 // 8 + 4096) * 5 // 4 + 4096
    counts = compare(recs, k, 20, 1, G)
    assert counts.n_trivial + counts.n_lmtig >= 0.9 * len(recs)


def test_text_past_a_gigabyte():
    """FASTA text of more than 256 blocks of the parser's scans (4 MiB each), where a thread of the second pass composes
    more than one block: long headers, and records that lie across every other block's edge."""
    block, blocks, k = 1 << 22, 262, 31
    rng = np.random.default_rng(83)
    text = np.full(block * blocks + 777, ord("x"), dtype=np.uint8)
    text[0] = ord(">")
    recs = []
    for j in range(1, blocks + 1):
        s = synth.random_seq(rng, int(rng.integers(k + 1, 400)))
        recs.append(s)
        piece = np.frombuffer(("\n" + s + "\n>h").encode(), dtype=np.uint8)
        at = j * block - (len(piece) // 2 if j % 2 else 5000)
        text[at:at + len(piece)] = piece
    host = cfgpu.PackedInput(recs, k)
    with cfgpu.Compactor(k, 20, 1, 16384) as cx:
        cx.submit_text_ptr(text.ctypes.data, text.nbytes)
        n_bases, words, _, frag_len = cx.input_copy()
    assert n_bases == host.p.n_bases and frag_len == [len(s) for s in recs]
    assert words == [host.p.words[i] for i in range((n_bases + 31) // 32)]
    host.close()


@pytest.mark.parametrize("k,sizes", [(127, (1025, 2047, 2048, 2049)), (63, (1025, 2048, 2049)), (31, (2049, 4096, 4097))])
@pytest.mark.parametrize("local_div", [4, 8])
def test_batch_largest_tables(k, sizes, local_div):
    """Jobs of one subgraph that fill a batch's largest one-CTA tables (4096 slots beyond k = 31, 8192 up to it), and
    one instance more."""
    jobs = [instances(np.random.default_rng(84 + n), n, k, 20) for n in sizes]
    info = check_batch(k, 20, 1, 1, jobs, tuning=dict(local_div=local_div))
    assert info.n_redone == 0
