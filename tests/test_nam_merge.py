"""The NAM merge on the GPU against the oracle at the sizes where its shape changes: reads whose
hit counts lie around every group size and bucket bound, with few NAMs (one chain), with a NAM a
hit (more than a warp's slots, then more than 256), and with repeats' many open NAMs whose sort
keys tie; in each sort order, mapped together and one at a time."""
import numpy as np
import pytest

from gpu_index_test_gb300 import abi, native
from oracle import oracle_py

HITS = (1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 96, 97, 127, 128, 129, 130, 191, 193, 255, 256, 257,
        300, 520, 800)
SHAPES = ("chain", "scattered", "repeat", "mixed")


def read_of(rng, n_hits, shape, k, rs, queries):
    """Appends entries and queries of one read with n_hits hits to the lists."""
    # runs of up to 90 entries a query (never filtered: the cutoff is 100)
    runs, left = [], n_hits
    most = {"chain": 1, "scattered": 30, "repeat": 90, "mixed": 40}[shape]
    while left:
        m = int(min(left, rng.integers(1, most + 1)))
        runs.append(m)
        left -= m
    if len(runs) > 1600:
        raise ValueError("too many queries for a read")
    fwd = len(runs) if shape == "chain" else int(rng.integers(0, len(runs) + 1))
    out = []
    for rc, part in ((0, runs[:fwd]), (1, runs[fwd:])):
        starts = np.sort(rng.choice(4000 if len(part) > 100 else 40 * max(1, len(part)), len(part), replace=False))
        for qs, m in zip(starts, part):
            span = int(rng.integers(k, k + 30))
            h = np.uint64(rng.integers(1 << 20, (1 << 63) - 1))
            if shape == "chain":
                pos = np.array([100000 + int(qs)])
            elif shape == "repeat":   # copies a short period apart, all open at once
                pos = 50000 + int(qs) + 6 * np.arange(m)
            elif shape == "scattered":
                pos = np.sort(rng.choice(30_000_000, m, replace=False))
            else:
                pos = np.unique(np.concatenate([[70000 + int(qs)], rng.choice(200_000, m)]))[:m]
            ref = 0 if shape == "repeat" else rng.integers(0, 3, len(pos))
            # a run keeps the entries of least length difference: all the same span
            for p, r in zip(pos, np.broadcast_to(ref, len(pos))):
                rs.append((h, int(p), (int(r) << 8) | (span - k)))
            out.append((h, int(qs), int(qs) + span, rc))
    queries.append(out)


@pytest.fixture(scope="module")
def merged():
    rng = np.random.default_rng(17)
    p = native.params_from_read_length(150)
    rs, queries = [(1, 0, 0)], []   # the smallest hash is never found
    for shape in SHAPES:
        for n in HITS:
            read_of(rng, n, shape, p.k, rs, queries)
    ent = np.array(rs, abi.REF_RANDSTROBE)
    ent = np.sort(ent, order=["hash", "position", "packed"])
    bits = 10
    starts = np.searchsorted(ent["hash"] >> np.uint64(64 - bits), np.arange((1 << bits) + 1, dtype=np.uint64)).astype(
        np.uint64)
    q = np.concatenate([np.array([(h, s, e, rc, 0) for h, s, e, rc in r],
                                 np.dtype([("hash", "<u8"), ("start", "<u4"), ("end", "<u4"), ("is_reverse", "u1"),
                                           ("_p", "u1")])) for r in queries])
    full = np.zeros(len(q), abi.QUERY_RANDSTROBE)
    for f in ("hash", "start", "end", "is_reverse"):
        full[f] = q[f]
    offs = np.concatenate([[0], np.cumsum([len(r) for r in queries])]).astype(np.uint64)
    return p, ent, starts, bits, full, offs


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [abi.GBSA_SORT_SCORE, abi.GBSA_SORT_REF_MATE1, abi.GBSA_SORT_REF_MATE2])
def test_merge_at_group_and_slot_bounds(merged, mode):
    p, ent, starts, bits, q, offs = merged
    o = oracle_py.Index.load(p, ent, starts, bits, 100)
    idx = native.Index.load(p, ent, starts, bits, 100)
    m = native.Mapper(idx, abi.map_options(sort_mode=mode), max_reads=256)
    nams, noff, _ = m.find_nams(q, offs)
    most = 0
    for i in range(len(offs) - 1):
        want, _ = o.find_nams(q[int(offs[i]): int(offs[i + 1])])
        want = oracle_py.sort_nams(want, mode)
        got = nams[int(noff[i]): int(noff[i + 1])]
        assert len(got) == len(want), i
        for f in abi.NAM_COMPARED:
            assert (got[f] == want[f]).all(), (i, f)
        most = max(most, len(want))
    assert most > 256   # the list in memory is reached too
    # each read alone gives the same
    for i in (0, len(HITS) + 5, 2 * len(HITS) - 1, 3 * len(HITS) - 2, 4 * len(HITS) - 1):
        one, _, _ = m.find_nams(q[int(offs[i]): int(offs[i + 1])], offs[i: i + 2] - offs[i])
        assert (one == nams[int(noff[i]): int(noff[i + 1])]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [abi.GBSA_SORT_SCORE, abi.GBSA_SORT_REF_MATE2])
@pytest.mark.parametrize("block", [0, 1])
def test_rescue_merge_and_sort_bounds(mode, block):
    """find_nams_rescue of reads whose NAM counts lie around the sorts' sizes (a warp's, a
    block's registers, a cluster's tiles, memory), with a warp and with a block a read: NAMs
    that join hits of many queries, NAMs that compete for hits, reference ids and query ends
    too wide for one key word, and two queries with the same start."""
    rng = np.random.default_rng(23)
    p = native.params_from_read_length(150)
    rs, reads = [(1, 0, 0)], []
    counts = (3, 31, 255, 256, 257, 511, 512, 513, 1000, 1025, 2047, 2048, 2049, 4096, 4097, 8192, 8193, 16384, 16500)

    def read(n, near, refs, wide, same_start):
        out, left, qs = [], n, 0
        while left:
            m = int(min(left, rng.integers(1, 1001)))
            left -= m
            span = int(rng.integers(p.k, p.k + 40))
            h = int(rng.integers(1 << 20, (1 << 62) - 1))
            pos = (np.sort(rng.choice(200_000_000, m, replace=False)) if not near
                   else 5000 + qs + near * np.arange(m) + rng.integers(0, 2))
            ref = rng.integers(0, refs, m)
            for x, r, s in zip(pos, ref, rng.integers(0, 3, m) + span):
                rs.append((h, int(x), (int(r) << 8) | (int(s) - p.k)))
            out.append((h, qs, qs + span, int(rng.integers(2))))
            qs += 0 if same_start and len(out) == 2 else int(rng.integers(1, 200 if wide else 9))
        reads.append(out)

    for n in counts:
        read(n, 0, 3, False, False)
    for near in (1, 2, 3, 6):
        for refs in (1, 2, 20):
            read(int(rng.integers(2000, 9000)), near, refs, False, False)
            read(int(rng.integers(40, 700)), near, refs, False, False)
    read(3000, 0, 1 << 24, True, False)
    read(700, 0, 1 << 24, True, False)
    read(3000, 2, 2, False, True)
    ent = np.sort(np.array(rs, abi.REF_RANDSTROBE), order=["hash", "position", "packed"])
    bits = 10
    starts = np.searchsorted(ent["hash"] >> np.uint64(64 - bits), np.arange((1 << bits) + 1, dtype=np.uint64)).astype(
        np.uint64)
    q = np.zeros(sum(len(r) for r in reads), abi.QUERY_RANDSTROBE)
    flat = [x for r in reads for x in r]
    for i, f in enumerate(("hash", "start", "end", "is_reverse")):
        q[f] = [x[i] for x in flat]
    offs = np.concatenate([[0], np.cumsum([len(r) for r in reads])]).astype(np.uint64)
    o = oracle_py.Index.load(p, ent, starts, bits, 100)
    m = native.Mapper(native.Index.load(p, ent, starts, bits, 100), abi.map_options(sort_mode=mode), max_reads=256)
    m.set_rescue_block(block)
    nams, noff, _ = m.find_nams(q, offs, rescue=True, rescue_cutoff=1500)
    for i in range(len(reads)):
        want = oracle_py.sort_nams(o.find_nams_rescue(q[int(offs[i]): int(offs[i + 1])], 1500), mode)
        got = nams[int(noff[i]): int(noff[i + 1])]
        assert len(got) == len(want), i
        for f in abi.NAM_COMPARED:
            assert (got[f] == want[f]).all(), (i, f)
