"""NAMs of one read that agree in everything the sort's one-word keys hold (score, orientation,
reference id, query interval, reference start) and differ in their reference ends: queries with
the same start and hash open equal NAMs, which then take different hits of a later query."""
import numpy as np
import pytest

from gpu_index_test_gb300 import abi, native
from oracle import oracle_py

K = 20


def equal_pair_read(n_others, copies):
    """Entries and queries of a read whose first NAMs tie that way, and n_others single hits."""
    rs, q = [(1, 0, 0)], []
    h0, h1 = np.uint64(11 << 40), np.uint64(12 << 40)
    for c in range(copies):   # each copy: NAMs at the same place of a reference of its own
        rs.append((h0, 1000, c << 8 | 60 - K))
        rs.append((h1, 1040, c << 8 | 70 - K))   # end 1110
        rs.append((h1, 1045, c << 8 | 50 - K))   # end 1095: the same score, 2 * (2 * min - max)
    q += [(h0, 0, 60, 0), (h0, 0, 60, 0), (h1, 50, 100, 0)]
    for i in range(0, n_others, 100):
        h = np.uint64((13 << 40) + i)
        rs += [(h, 50_000 + 100 * j, 7 << 8) for j in range(i, min(i + 100, n_others))]
        q.append((h, 200 + i, 220 + i, 0))
    ent = np.sort(np.array(rs, abi.REF_RANDSTROBE), order=["hash", "position", "packed"])
    queries = np.zeros(len(q), abi.QUERY_RANDSTROBE)
    for i, f in enumerate(("hash", "start", "end", "is_reverse")):
        queries[f] = [x[i] for x in q]
    return ent, queries


@pytest.mark.parametrize("copies", [1, 2])
def test_the_oracle_orders_them_by_their_ends(copies):
    ent, q = equal_pair_read(300, copies)
    p = oracle_py.params_from_read_length(150)
    assert p.k == K
    o = oracle_py.Index.load(p, ent, starts_of(ent), 10, 1000)
    got = oracle_py.sort_nams(o.find_nams(q)[0])[:2 * copies]
    assert (got["score"] == 180).all() and (got["ref_start"] == 1000).all() and (got["query_end"] == 100).all()
    assert got["ref_end"].tolist() == [1095, 1110] * copies


def starts_of(ent, bits=10):
    return np.searchsorted(ent["hash"] >> np.uint64(64 - bits), np.arange((1 << bits) + 1, dtype=np.uint64)).astype(
        np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("rescue", [False, True])
@pytest.mark.parametrize("copies", [1, 2])
@pytest.mark.parametrize("n_others", [10, 120, 300, 900])
def test_ties_by_the_reference_end(n_others, copies, rescue):
    """In registers, in the block merge's sort and in the sort of rescued reads."""
    ent, q = equal_pair_read(n_others, copies)
    p = native.params_from_read_length(150)
    o = oracle_py.Index.load(p, ent, starts_of(ent), 10, 1000)
    idx = native.Index.load(p, ent, starts_of(ent), 10, 1000)
    m = native.Mapper(idx, max_reads=16)
    got = m.find_nams(q, np.array([0, len(q)], np.uint64), rescue=rescue, rescue_cutoff=1000)[0]
    want = oracle_py.sort_nams(o.find_nams_rescue(q, 1000) if rescue else o.find_nams(q)[0])
    assert len(got) == len(want) == 2 * copies + n_others
    for f in abi.NAM_COMPARED:
        assert (got[f] == want[f]).all(), f
