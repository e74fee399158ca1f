"""Arena room that warps take ahead in pieces: a batch whose hits fit the arena does not outgrow it
because of what is left of the pieces, whatever share of a piece a read's hits are."""
import numpy as np
import pytest

from golden_cases import nams_equal
from gpu_index_test_gb300 import native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [3, 4, 5, 6])
def test_hits_of_a_third_of_a_piece(copies):
    """A genome in `copies` copies: 25 hits a read and copy.  The arena holds 166 a read."""
    g = synth.make_genome(synth.GenomeParams(seed=8, total_len=400_000, n_contigs=2))
    rng = np.random.default_rng(1)
    s = np.concatenate([g.seq] * copies)
    k = np.flatnonzero(rng.random(s.size) < 0.002)
    s[k] = rng.choice(np.frombuffer(b"ACGT", np.uint8), len(k))
    g = synth.Genome(s, np.tile(g.lengths, copies),
                     np.concatenate([g.offsets + np.uint64(400_000 * i) for i in range(copies)]))
    p = native.params_from_read_length(150)
    idx, o = native.Index.build(p, g), oracle_py.Index.build(oracle_py.params_from_read_length(150), g)
    n = 300_000
    reads = synth.make_reads(g, synth.ReadParams(seed=9, n_units=n, sub=(0.002, 0.002), indel_rate=0.0))
    m = native.Mapper(idx, max_reads=n, max_bases=int(reads.seq.size))
    m.set_pipeline(1)
    x = m.map_reads(reads, capacity=(copies + 4) * n)
    hits = m.last_counts()["hits"]
    assert 20 * copies * n < hits < 0.95 * 166 * n and m.retries() == 0, hits / n
    some = reads.subset(np.arange(0, n, 300))
    y = o.map_reads(some, n_threads=8)
    at = x[1].astype(np.int64)
    assert nams_equal(np.concatenate([x[0][at[i]: at[i + 1]] for i in range(0, n, 300)]), y[0])
