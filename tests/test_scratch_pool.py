"""Scratch of the calls that allocate: the same results from several threads at once, with and
without an index alive, bounded between calls and given back with the last index."""
import gc
import threading

import numpy as np
import pytest

from gpu_index_test_gb300 import native, synth

pytestmark = pytest.mark.gpu


def test_threads_bounds_and_return():
    import torch

    gc.collect()
    g = synth.make_genome(synth.GenomeParams(seed=1, total_len=500_000, n_contigs=2))
    sets = [synth.make_reads(g, synth.ReadParams(seed=s, n_units=n, len_min=60, len_max=700, paired_frac=0.0))
            for s, n in ((2, 300), (3, 20_000), (4, 5_000), (5, 60_000))]
    p = native.params_from_read_length(150)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    alone = [native.randstrobes_query(p, r) for r in sets]          # no index of ours
    for kept in (True, False):
        idx = native.Index.build(p, g) if kept else None
        got, errors = [[] for _ in sets], []

        def run(i):
            try:
                for _ in range(6):
                    got[i].append(native.randstrobes_query(p, sets[i]))
                native.Index.build(p, g).free()
            except Exception as e:   # noqa: BLE001 (reported below)
                errors.append(e)

        threads = [threading.Thread(target=run, args=(i,)) for i in range(len(sets))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors
        for want, runs in zip(alone, got):
            for q, off in runs:
                assert (off == want[1]).all()
                for f in ("hash", "start", "end", "is_reverse"):
                    assert (q[f] == want[0][f]).all()
        torch.cuda.synchronize()
        slack = 128 << 20   # contexts' and streams' own memory
        assert torch.cuda.mem_get_info()[0] >= before - (256 << 20) - slack - (16 << 20)
        if idx is not None:
            idx.free()
    assert torch.cuda.mem_get_info()[0] >= before - slack
