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
