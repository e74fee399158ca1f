"""Large batches of reads that are not clean (an N, a U, a tied window) or have more queries than
the one-go seeding holds: the arenas that hold a batch of clean reads hold them too, and the
results are the oracle's."""
import numpy as np
import pytest
import torch

from golden_cases import nams_equal
from gpu_index_test_gb300 import native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu
N = 120_000


@pytest.fixture(scope="module")
def made():
    g = synth.make_genome(synth.GenomeParams(seed=31, total_len=2_000_000, n_contigs=2))
    p = native.params_from_read_length(150)
    idx, o = native.Index.build(p, g), oracle_py.Index.build(oracle_py.params_from_read_length(150), g)
    return g, p, idx, o, synth.make_reads(g, synth.ReadParams(seed=32, n_units=N // 2, paired_frac=1.0))


def changed(reads, form):
    rng = np.random.default_rng(5)
    seq = reads.seq.copy()
    if form == "N":
        seq[reads.offsets.astype(np.int64) + rng.integers(0, 150, reads.n)] = ord("N")
    elif form == "U":
        seq[seq == ord("T")] = ord("U")
    elif form == "tied":   # a stretch of one base near an end
        for i in range(30):
            seq[reads.offsets.astype(np.int64) + i] = ord("A")
    return synth.Reads(seq, reads.offsets, reads.lengths)


def mapped_as_the_oracle(x, o, reads, step):
    some = reads.subset(np.arange(0, reads.n, step))
    y = o.map_reads(some, n_threads=8)
    at = x[1].astype(np.int64)
    got = np.concatenate([x[0][at[i]: at[i + 1]] for i in range(0, reads.n, step)])
    assert (np.diff(at)[::step] == np.diff(y[1].astype(np.int64))).all() and nams_equal(got, y[0])
    assert (x[2][::step] == y[2]).all() and (x[3][::step] == y[3]).all()


def test_reads_of_many_queries(made):
    """450 bases and syncmers of three s-mers: 270 queries a read, which go by the steps.  The
    query arena holds 233 a read at first: it grows once, to what they use."""
    g = made[0]
    p = native.params_make(150, 20, 18, 1, 7, 255, 80)
    idx, o = native.Index.build(p, g), oracle_py.Index.build(p, g)
    reads = synth.make_reads(g, synth.ReadParams(seed=33, n_units=60_000, len_min=450, len_max=450))
    m = native.Mapper(idx, max_reads=reads.n, max_bases=int(reads.seq.size))
    x = m.map_reads(reads, capacity=32 * reads.n)
    assert m.retries() == 1 and m.last_counts()["long_reads"] < reads.n // 10
    mapped_as_the_oracle(x, o, reads, 60)


@pytest.mark.parametrize("form", ["clean", "N", "U", "tied"])
def test_a_batch_of_them_fits(made, form):
    g, p, idx, o, clean = made
    reads = changed(clean, form)
    m = native.Mapper(idx, max_reads=N, max_bases=int(reads.seq.size))
    x = m.map_reads(reads, capacity=16 * N)
    assert m.retries() == 0
    mapped_as_the_oracle(x, o, reads, 30)
    # the batched form: one eager run, then the graph
    at = x[1].astype(np.int64)
    b = native.Batcher(idx, max_reads=N, max_bases=int(reads.seq.size))
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
    d = [up(reads.seq), up(reads.offsets), up(reads.lengths)]
    nams = torch.zeros(16 * N * 11, dtype=torch.int32, device="cuda")
    off = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    for _ in range(2):
        total = b.map_reads_device(*[t.data_ptr() for t in d], N, nams.data_ptr(), 16 * N, off.data_ptr())
        assert total == len(x[0]) and (off.cpu().numpy() == at).all()
    assert b.stats()["eager_runs"] == 1 and b.stats()["graph_launches"] == 1
    assert nams_equal(nams.cpu().numpy()[: 11 * total].view(x[0].dtype), x[0])
