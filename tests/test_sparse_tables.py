"""Bucket tables with few entries for their buckets, with about as many, and with hundreds a
bucket: built, loaded, searched and mapped against, compared with the oracle; and what a table
mostly of empty buckets costs to build beside loading it."""
import time

import numpy as np
import pytest
import torch

from golden_cases import nams_equal
from gpu_index_test_gb300 import native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu


def genome_of(n, seed):
    seq = np.random.default_rng(seed).choice(np.frombuffer(b"ACGT", np.uint8), n).astype(np.uint8)
    return synth.Genome(seq, np.array([n], np.uint64), np.zeros(1, np.uint64))


@pytest.mark.parametrize("bits", [8, 11, 13, 16, 20])
@pytest.mark.parametrize("n", [100, 200, 3000, 30_000, 400_000])
def test_tables_of_all_densities(n, bits):
    g = genome_of(n, n + bits)
    p, op = native.params_from_read_length(150), oracle_py.params_from_read_length(150)
    idx, o = native.Index.build(p, g, bits=bits), oracle_py.Index.build(op, g, bits=bits)
    rs, st = idx.export()
    assert (rs == o.randstrobes()).all() and (st == o.starts()).all()
    reads = synth.make_reads(g, synth.ReadParams(seed=3, n_units=200, len_min=min(150, n), len_max=min(150, n)))
    y = o.map_reads(reads, n_threads=4)
    for i in (idx, native.Index.load(p, rs, st, bits, idx.info().filter_cutoff)):
        x = native.Mapper(i, max_reads=256).map_reads(reads)
        assert (x[1] == y[1]).all() and (x[2] == y[2]).all() and (x[3] == y[3]).all() and nams_equal(x[0], y[0])


def test_what_empty_buckets_cost():
    """13 entries in 2^24 buckets: their spans written by one thread each took 200 times as long
    as loading the table (400 MB of them on the device), now 6 times."""
    g, p = genome_of(100, 1), native.params_from_read_length(150)
    idx = native.Index.build(p, g, bits=24)
    rs, st = idx.export()

    def best(f):
        out = []
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            f()
            torch.cuda.synchronize()
            out.append(time.perf_counter() - t)
        return min(out)

    assert best(lambda: native.Index.build(p, g, bits=24)) < 40 * best(lambda: native.Index.load(p, rs, st, 24, 30))
