"""find_nams on long reads with more NAMs than the register merge has slots (128) and few of them
open at a time, against the oracle: around the number of open NAMs that the slots take over
(96), across the orientations, with NAMs that tie and NAMs that live through the whole read,
some of them among reads of other kinds; and what long reads cost beside seeding them."""
import numpy as np
import pytest

from gpu_index_test_gb300 import abi, native, synth
from oracle import oracle_py

K, BITS = 20, 10


def read_of(rng, shape, entries):
    """Queries of one read; appends their entries."""
    step, span, hits, n = {           # about span / step queries are open at a time
        "sparse": (9, 40, 1, 420), "pairs": (9, 60, 2, 420), "dense": (2, 47, 4, 400), "full": (2, 49, 4, 400),
        "over": (2, 80, 4, 300), "short": (30, 25, 1, 129), "slots": (30, 25, 1, 128), "ties": (12, 50, 3, 300),
        "lived": (9, 40, 1, 420), "deep": (1, 30, 3, 1500)}[shape]
    out = []
    fwd = int(rng.integers(0, n + 1)) if shape not in ("dense", "full") else n
    for rc, m in ((0, fwd), (1, n - fwd)):
        for i in range(m):
            qs, h = i * step, int(rng.integers(1 << 20, (1 << 63) - 1))
            e = span + int(rng.integers(0, 1 if shape in ("dense", "full", "ties") else 12))
            if shape == "ties":      # copies on references of their own, in runs of one position
                at = [(1000 + qs // 24 * 90, r) for r in range(hits)]
            else:
                at = [(int(x), int(rng.integers(0, 3))) for x in np.sort(rng.choice(40_000_000, hits, replace=False))]
            if shape == "lived":     # a chain that takes a hit of every query
                at = sorted(at + [(50_000_000 + qs, 1)])
            entries += [(h, x, (r << 8) | (e - K)) for x, r in sorted(at)]
            out.append((h, qs, qs + e, rc))
    return out


SHAPES = ("sparse", "pairs", "dense", "full", "over", "short", "slots", "ties", "lived", "deep")


@pytest.fixture(scope="module")
def made():
    rng = np.random.default_rng(41)
    entries, reads = [(1, 0, 0)], []
    for shape in SHAPES * 3:
        reads.append(read_of(rng, shape, entries))
    ent = np.sort(np.array(entries, abi.REF_RANDSTROBE), order=["hash", "position", "packed"])
    starts = np.searchsorted(ent["hash"] >> np.uint64(64 - BITS),
                             np.arange((1 << BITS) + 1, dtype=np.uint64)).astype(np.uint64)
    q = np.zeros(sum(map(len, reads)), abi.QUERY_RANDSTROBE)
    for i, f in enumerate(("hash", "start", "end", "is_reverse")):
        q[f] = [x[i] for r in reads for x in r]
    return ent, starts, q, np.concatenate([[0], np.cumsum([len(r) for r in reads])]).astype(np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [abi.GBSA_SORT_SCORE, abi.GBSA_SORT_REF_MATE1, abi.GBSA_SORT_REF_MATE2])
def test_many_nams_few_open(made, mode):
    ent, starts, q, offs = made
    p = native.params_from_read_length(150)
    assert p.k == K
    o = oracle_py.Index.load(p, ent, starts, BITS, 100)
    m = native.Mapper(native.Index.load(p, ent, starts, BITS, 100), abi.map_options(sort_mode=mode), max_reads=64)
    nams, noff, _ = m.find_nams(q, offs)
    for i in range(len(offs) - 1):
        want = oracle_py.sort_nams(o.find_nams(q[int(offs[i]): int(offs[i + 1])])[0], mode)
        got = nams[int(noff[i]): int(noff[i + 1])]
        assert len(got) == len(want), (i, SHAPES[i % len(SHAPES)])
        for f in abi.NAM_COMPARED:
            assert (got[f] == want[f]).all(), (i, f)
        one, _, _ = m.find_nams(q[int(offs[i]): int(offs[i + 1])], offs[i: i + 2] - offs[i])
        assert (one == got).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n, times", [(100, 12), (2000, 6)])
def test_what_their_nams_cost_beside_their_seeds(n, times):
    """Reads of 4,000 bp, most with more NAMs than slots: merged by a block each, query by query,
    this took 36 and 11 times as long as the seeding, now 4 and 2 times."""
    g = synth.make_genome(synth.genome_params("C2", scale=0.2, seed=1))
    p = native.params_from_read_length(400)
    idx, o = native.Index.build(p, g), oracle_py.Index.build(oracle_py.params_from_read_length(400), g)
    reads = synth.make_reads(g, synth.ReadParams(seed=7, n_units=n, len_min=4000, len_max=4000))
    m = native.Mapper(idx, max_reads=n, max_bases=int(reads.seq.size))
    m.set_profile(True)
    stages = []
    for _ in range(4):
        x = m.map_reads(reads, capacity=400 * n)
        stages.append(m.stage_ms())
    some = reads.subset(np.arange(0, n, n // 50))
    y = o.map_reads(some, n_threads=8)
    at = x[1].astype(np.int64)
    got = np.concatenate([x[0][at[i]: at[i + 1]] for i in range(0, n, n // 50)])
    assert len(got) == len(y[0]) and all((got[f] == y[0][f]).all() for f in abi.NAM_COMPARED)
    assert min(s["nams"] + s["nams_warp"] for s in stages) < times * min(s["seed_long"] for s in stages)
