"""Loaded tables whose start indices stop short of the last entry: the last used bucket ends
inside a run of equal hashes, or with its last entry, and every later bucket is empty.  The run's
walk goes on behind the bucket's end, so what a query's hits are counted as and what is written
have to agree."""
import numpy as np
import pytest

from golden_cases import nams_equal
from gpu_index_test_gb300 import abi, native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu


def reads_of(rng, n):
    lens = np.full(n, 150, np.uint32)
    return synth.Reads(rng.choice(np.frombuffer(b"ACGT", np.uint8), 150 * n).astype(np.uint8),
                       np.arange(n, dtype=np.uint64) * np.uint64(150), lens)


def table(rng, hashes, bits, run):
    """`run` entries of every hash, positions rising, and one smaller hash in front."""
    rs = [(1, 0, 0)]
    for h in hashes:
        rs += [(int(h), int(x), int(rng.integers(0, 3)) << 8 | 30)
               for x in np.sort(rng.choice(1 << 20, run, replace=False))]
    ent = np.sort(np.array(rs, abi.REF_RANDSTROBE), order=["hash", "position", "packed"])
    starts = np.searchsorted(ent["hash"] >> np.uint64(64 - bits), np.arange((1 << bits) + 1, dtype=np.uint64))
    return ent, starts.astype(np.uint64)


@pytest.mark.parametrize("run", [1, 2, 8, 30])
@pytest.mark.parametrize("bits", [8, 14])
def test_starts_that_stop_short(run, bits):
    rng = np.random.default_rng(run)
    p, op = native.params_from_read_length(150), oracle_py.params_from_read_length(150)
    reads = reads_of(rng, 200)
    q = native.randstrobes_query(p, reads)[0]
    hashes = np.unique(q["hash"][rng.random(len(q)) < 0.7])
    ent, starts = table(rng, hashes, bits, run)
    n = len(ent)
    h = ent["hash"][n // 2:]
    # cuts inside a run and between two buckets
    top = h >> np.uint64(64 - bits)
    cuts = [np.flatnonzero(top[1:] != top[:-1])] + ([np.flatnonzero(h[1:] == h[:-1])] if run > 1 else [])
    for cut in (n // 2 + 1 + int(at[x]) for at in cuts for x in (0, len(at) // 2, -1)):
        short = np.minimum(starts, np.uint64(cut))
        idx, o = native.Index.load(p, ent, short, bits, 100), oracle_py.Index.load(op, ent, short, bits, 100)
        assert (idx.find(ent["hash"]) == np.array([o.find(int(x)) for x in ent["hash"]], np.uint64)).all()
        y = o.map_reads(reads, n_threads=4)
        m = native.Mapper(idx, max_reads=256)
        for fuse in (None, 0):
            if fuse is not None:
                m.set_fuse_limit(fuse)
            x = m.map_reads(reads)
            assert (x[1] == y[1]).all() and (x[2] == y[2]).all() and (x[3] == y[3]).all() and nams_equal(x[0], y[0])
        x = native.Batcher(idx, max_reads=256).map_reads(reads)
        assert (x[1] == y[1]).all() and nams_equal(x[0], y[0])
