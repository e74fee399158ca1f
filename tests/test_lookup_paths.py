"""Seeding and lookup in one go (clean reads, tagged buckets) against the oracle and against the
path by steps, at the sizes and forms where the two part: bucket sizes around the four tags,
runs and the filter cutoff, tags that agree by chance, tables out of order; reads with N, lower
case and U, tied windows, every alignment, and lengths around the chunk, query and buffer sizes."""
import numpy as np
import pytest

from golden_cases import nams_equal
from gpu_index_test_gb300 import abi, native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu


def same(a, b):
    return (a[1] == b[1]).all() and (a[2] == b[2]).all() and (a[3] == b[3]).all() and nams_equal(a[0], b[0])


def reads_of(seqs):
    lens = np.array([len(s) for s in seqs], np.uint32)
    offs = np.concatenate([[0], np.cumsum(lens[:-1])]).astype(np.uint64)
    return synth.Reads(np.frombuffer(b"".join(seqs), np.uint8).copy(), offs, lens)


def odd_reads(rng, genome, p):
    """Reads cut from the genome, at lengths around the limits, some changed."""
    rc = bytes.maketrans(b"ACGTacgtN", b"TGCAtgcaN")
    lengths = [1, p.k - 1, p.k, p.k + 1, 31, 32, 33, 50, 51, 52, 63, 64, 65, 83, 84, 100, 127, 128, 129, 150, 151, 250,
               251, 255, 256, 257, 300, 383, 384, 385, 447, 448, 449, 500, 511, 512, 513, 600, 1000, 2100]
    out = []
    for n in lengths:
        for form in range(8):
            at = int(rng.integers(0, len(genome) - n))
            s = bytearray(genome[at: at + n])
            if rng.random() < 0.5:
                s = bytearray(bytes(s).translate(rc)[::-1])
            for _ in range(int(rng.integers(0, 3))):   # sequencing errors
                s[int(rng.integers(0, n))] = b"ACGT"[int(rng.integers(0, 4))]
            if form == 1:
                s[int(rng.integers(0, n))] = ord("N")
            elif form == 2:
                s[n - 1] = ord("n")
            elif form == 3:
                s = bytearray(bytes(s).lower())
            elif form == 4:
                s = bytearray(bytes(s).replace(b"T", b"U"))
            elif form == 5 and n > 40:   # tied windows at a place
                b = int(rng.integers(0, n - 40))
                s[b: b + 40] = (b"ACACACACAC" * 4, b"A" * 40, b"ACGT" * 10)[int(rng.integers(0, 3))]
            elif form == 6:
                s[0] = b"*R\x00\xc1"[int(rng.integers(0, 4))]
            out.append(bytes(s))
    return out


@pytest.mark.parametrize("r", [50, 75, 100, 125, 150, 250, 400])
def test_reads_at_the_limits(r):
    rng = np.random.default_rng(r)
    g = synth.make_genome(synth.GenomeParams(seed=r, total_len=300_000, n_contigs=2, dup_frac=0.05, str_frac=0.02))
    p = native.params_from_read_length(r)
    idx = native.Index.build(p, g)
    o = oracle_py.Index.build(oracle_py.params_from_read_length(r), g)
    genome = g.seq.tobytes()
    reads = reads_of(odd_reads(rng, genome, p))
    y = o.map_reads(reads, n_threads=8)
    m = native.Mapper(idx)
    assert same(m.map_reads(reads), y)
    assert m.fused_lookup()
    m.set_fuse_limit(0)
    assert same(m.map_reads(reads), y)
    assert same(native.Batcher(idx, max_reads=reads.n).map_reads(reads), y)


@pytest.mark.parametrize("k,s,l,u,q,dist", [(20, 16, 1, 7, 255, 80), (20, 16, 0, 0, 511, 80), (22, 18, 2, 12, 127, 255),
                                            (30, 12, 1, 5, 255, 120), (32, 30, 1, 7, 255, 255), (9, 1, 1, 3, 15, 60)])
def test_parameters_of_either_path(k, s, l, u, q, dist):
    """Parameters that the profiles do not use: windows of 3 to 19 s-mers, s over 16, selection
    bits wider than a byte (the path by steps)."""
    rng = np.random.default_rng(k)
    g = synth.make_genome(synth.GenomeParams(seed=5, total_len=100_000, n_contigs=2, dup_frac=0.05, str_frac=0.02))
    p = native.params_make(150, k, s, l, u, q, dist)
    idx, o = native.Index.build(p, g), oracle_py.Index.build(p, g)
    genome = g.seq.tobytes()
    reads = reads_of(odd_reads(rng, genome, p))
    assert same(native.Mapper(idx).map_reads(reads), o.map_reads(reads, n_threads=8))


def table(rng, query_hashes, bits, late=False):
    """Entries for the queries' hashes in runs of 1 to 9 and around the cutoff of 30, and others
    beside them: in the same bucket, and there with the same tag."""
    out = []
    for h in query_hashes:
        h = int(h)
        n = int(rng.choice([1, 1, 1, 2, 3, 4, 5, 9, 29, 30, 31, 60]))
        for pos in np.sort(rng.choice(1 << 20, n, replace=False)):
            out.append((h, int(pos), int(rng.integers(0, 3)) << 8 | int(rng.integers(0, 90))))
        for _ in range(int(rng.integers(0, 6))):
            low = int(rng.integers(0, 1 << 24))
            near = (h >> 24 << 24) | low                                      # same bucket, same tag
            far = (h >> (64 - bits) << (64 - bits)) | int(rng.integers(0, 1 << (64 - bits)))   # same bucket
            out.append(((near, far)[int(rng.integers(0, 2))], int(rng.integers(0, 1 << 20)), 7))
    ent = np.sort(np.array(out + [(1, 0, 0)], abi.REF_RANDSTROBE), order=["hash", "position", "packed"])
    starts = np.searchsorted(ent["hash"] >> np.uint64(64 - bits), np.arange((1 << bits) + 1, dtype=np.uint64)).astype(
        np.uint64)
    if late:       # entries out of order within a bucket
        for b in np.flatnonzero(np.diff(starts) == 3):
            a = int(starts[b])
            ent[a: a + 3] = ent[a: a + 3][::-1]
    return ent, starts


@pytest.mark.parametrize("cutoff", [1, 2, 30, 100, 255, 256, 1000])
def test_bucket_forms(cutoff):
    rng = np.random.default_rng(cutoff)
    p, op = native.params_from_read_length(150), oracle_py.params_from_read_length(150)
    seqs = [bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 150)) for _ in range(300)]
    reads = reads_of(seqs)
    q = native.randstrobes_query(p, reads)[0]
    hashes = np.unique(q["hash"][rng.random(len(q)) < 0.6])
    for bits in (8, 12, 20):
        ent, starts = table(rng, hashes, bits)
        idx, o = native.Index.load(p, ent, starts, bits, cutoff), oracle_py.Index.load(op, ent, starts, bits, cutoff)
        m = native.Mapper(idx, max_reads=1024)
        y = o.map_reads(reads, n_threads=4)
        assert y[1][-1] > 0
        assert same(m.map_reads(reads), y)
        m.set_fuse_limit(0)
        assert same(m.map_reads(reads), y)


def test_a_table_out_of_order_is_searched_in_order():
    rng = np.random.default_rng(3)
    p, op = native.params_from_read_length(150), oracle_py.params_from_read_length(150)
    reads = reads_of([bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), 150)) for _ in range(100)])
    q = native.randstrobes_query(p, reads)[0]
    ent, starts = table(rng, np.unique(q["hash"]), 12, late=True)
    idx, o = native.Index.load(p, ent, starts, 12, 30), oracle_py.Index.load(op, ent, starts, 12, 30)
    h = ent["hash"]
    assert (idx.find(h) == np.array([o.find(int(x)) for x in h], np.uint64)).all()
    assert same(native.Mapper(idx, max_reads=1024).map_reads(reads), o.map_reads(reads, n_threads=4))


@pytest.mark.parametrize("rescue", [False, True])
def test_find_nams_takes_queries_in_any_order(rescue):
    """Reads' queries in order, shuffled, orientations mixed, none, one, and more than a warp
    ranks (1,024) in and out of order; offsets that do not begin at 0."""
    rng = np.random.default_rng(11)
    g = synth.make_genome(synth.GenomeParams(seed=11, total_len=200_000, n_contigs=2, dup_frac=0.1))
    p = native.params_from_read_length(150)
    idx, o = native.Index.build(p, g), oracle_py.Index.build(oracle_py.params_from_read_length(150), g)
    genome = g.seq.tobytes()
    lens = [150, 150, 30, 300, 2600, 2600, 3000, 4000, 150, 20, 4000]
    q, off = native.randstrobes_query(p, reads_of([genome[a: a + n] for a, n in zip(range(500, 90_000, 7000), lens)]))
    q, off = q.copy(), off.copy()
    for r in range(len(lens)):
        a, b = int(off[r]), int(off[r + 1])
        if r in (1, 3, 5, 6, 7):
            q[a:b] = q[a:b][rng.permutation(b - a)]
        if r == 1 and b - a > 4:   # equal starts keep their order
            q["start"][a + 1: a + 3] = q["start"][a]
            q["end"][a + 1: a + 3] = q["end"][a]
    assert max(np.diff(off.astype(np.int64))) > 1024
    laid = q.copy()   # forward first, then by start, stable
    for r in range(len(lens)):
        part = q[int(off[r]): int(off[r + 1])]
        laid[int(off[r]): int(off[r + 1])] = part[np.lexsort((part["start"], part["is_reverse"] != 0))]
    for lo in (0, 1, 8):   # (the last: all in order)
        m = native.Mapper(idx, max_reads=64)
        a = m.find_nams(q, off[lo:], rescue=rescue, rescue_cutoff=50)
        b = m.find_nams(laid, off[lo:], rescue=rescue, rescue_cutoff=50)
        assert all((x == y).all() for x, y in zip(a, b))
        for i in range(2, len(lens) - lo):
            part = q[int(off[lo + i]): int(off[lo + i + 1])]
            want = o.find_nams_rescue(part, 50) if rescue else o.find_nams(part)[0]
            assert nams_equal(a[0][int(a[1][i]): int(a[1][i + 1])], oracle_py.sort_nams(want)), (lo, i)
