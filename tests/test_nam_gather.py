"""The gather of the NAM records at the sizes where its shape changes: batches around one read a
warp, a group of reads and the warps of a grid, reads with no NAMs, reads whose records stand
alone between rescued ones, and an output that ends within a group."""
import numpy as np
import pytest

from golden_cases import nams_equal
from gpu_index_test_gb300 import abi, native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def repeats():
    """A genome half of which is copies, so that many reads are rescued, and reads of which some
    are foreign to it."""
    rng = np.random.default_rng(8)
    bases = np.frombuffer(b"ACGT", np.uint8)
    unit = rng.choice(bases, 1500)
    parts = []
    for _ in range(130):   # more copies than the filter cutoff's most, 100
        parts += [unit, rng.choice(bases, 1500)]
    seq = np.concatenate(parts)
    g = synth.Genome(seq, np.array([len(seq)], np.uint64), np.array([0], np.uint64))
    n = 45_000
    reads = np.empty((n, 150), np.uint8)
    for i, at in enumerate(rng.integers(0, len(seq) - 150, n)):
        reads[i] = seq[at: at + 150] if i % 7 else rng.choice(bases, 150)
    reads = synth.Reads(reads.ravel(), 150 * np.arange(n, dtype=np.uint64), np.full(n, 150, np.uint32))
    p = native.params_from_read_length(150)
    return native.Index.build(p, g), oracle_py.Index.build(oracle_py.params_from_read_length(150), g), reads


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1000, 19_456, 19_457, 38_912, 45_000])
def test_batch_sizes(repeats, n):
    idx, o, reads = repeats
    part = reads.subset(np.arange(n))
    y = o.map_reads(part, n_threads=8)
    for x in (native.Mapper(idx, max_reads=n).map_reads(part), native.Batcher(idx, max_reads=n).map_reads(part)):
        assert (x[1] == y[1]).all() and (x[2] == y[2]).all() and (x[3] == y[3]).all()
        assert nams_equal(x[0], y[0])
    if n == 45_000:
        count = np.diff(y[1].astype(np.int64))
        assert (count == 0).any() and (count[y[3] != 0] > 0).any() and (count[y[3] == 0] > 0).any()


def test_an_output_that_ends_within_a_group(repeats):
    import torch

    idx, _, reads = repeats
    part = reads.subset(np.arange(2000))
    m = native.Mapper(idx, max_reads=2000)
    nams, offs, _, _ = m.map_reads(part)
    d = [torch.from_numpy(a.copy()).cuda() for a in (part.seq, part.offsets.view(np.int64), part.lengths.view(np.int32))]
    words = abi.NAM.itemsize // 4
    for cap in (0, 1, 31, 33, int(offs[1000]) + 1, len(nams) - 1):
        out = torch.full((words * (len(nams) + 64),), 7, dtype=torch.int32, device="cuda")
        d_offs = torch.zeros(2001, dtype=torch.int64, device="cuda")
        total = m.map_reads_device(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), 2000, out.data_ptr(), cap,
                                   d_offs.data_ptr())
        assert total == len(nams)
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert (got[words * cap:] == 7).all()
