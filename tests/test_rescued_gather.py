"""The gather of rescued reads against the oracle: batches of fewer and of more of them than the
grid has blocks and warps, with no NAMs, with lists for a warp (64) and with lists for the block
beside each other."""
import numpy as np
import pytest

from gpu_index_test_gb300 import abi, native
from oracle import oracle_py

COUNTS = (0, 1, 31, 32, 33, 63, 64, 65, 96, 255, 256, 257, 700)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 13, 300, 2433, 4000, 20_000])
def test_list_lengths(n):
    rng = np.random.default_rng(n)
    p = native.params_from_read_length(150)
    hashes = np.sort(rng.integers(1 << 40, (1 << 63) - 1, len(COUNTS)).astype(np.uint64))
    ent = np.array([(1, 0, 0)] + [(h, 10 + 1000 * j, 0) for h, c in zip(hashes, COUNTS) for j in range(c)],
                   abi.REF_RANDSTROBE)
    starts = np.searchsorted(ent["hash"] >> np.uint64(54), np.arange(1025, dtype=np.uint64)).astype(np.uint64)
    # a read in 40 with a long list, so that the result stays small
    kind = np.where(rng.random(n) < 0.025, rng.integers(0, len(COUNTS), n), rng.integers(0, 3, n))
    kind[0] = len(COUNTS) - 1
    q = np.zeros(n, abi.QUERY_RANDSTROBE)
    q["hash"], q["end"] = hashes[kind], p.k
    o = oracle_py.Index.load(p, ent, starts, 10, 1000)
    m = native.Mapper(native.Index.load(p, ent, starts, 10, 1000), max_reads=n)
    nams, offs, _ = m.find_nams(q, np.arange(n + 1, dtype=np.uint64), rescue=True, rescue_cutoff=1000)
    assert (np.diff(offs.astype(np.int64)) == np.array(COUNTS)[kind]).all()
    for k in range(len(COUNTS)):
        want = oracle_py.sort_nams(o.find_nams_rescue(q[kind == k][:1], 1000)) if (kind == k).any() else []
        for i in np.nonzero(kind == k)[0]:
            got = nams[int(offs[i]): int(offs[i + 1])]
            assert all((got[f] == want[f]).all() for f in abi.NAM_COMPARED)
