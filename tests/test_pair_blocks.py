"""NAM-pair scoring and planning of pairs with long NAM lists (reads in repeats) on the GPU
against the oracle, record by record: list lengths around the warp's 32 and around 32 blocks of
32, several reference ids, lists in and out of the sort order, ties in every compared field, and
more tries than a warp has lanes."""
import numpy as np
import pytest

from gpu_index_test_gb300 import abi, native
from oracle import oracle_py

SIZES = (0, 1, 2, 31, 32, 33, 64, 65, 97, 130, 700, 1055, 1400)


def make_list(rng, n, n_refs, spread, mate1, shuffle):
    a = np.zeros(n, abi.NAM)
    a["ref_id"] = rng.integers(0, n_refs, n) * 7
    a["is_rc"] = rng.integers(0, 2, n)
    a["query_start"] = rng.integers(0, 60, n)
    a["query_end"] = a["query_start"] + rng.integers(20, 60, n)
    a["ref_start"] = rng.integers(0, spread, n)
    a["ref_end"] = a["ref_start"] + rng.integers(20, 60, n)
    # hit counts as a repeat gives them: mostly low, a few high, many equal
    a["n_hits"] = np.minimum(1 + rng.geometric(0.3, n), 40)
    a["score"] = (a["n_hits"] * rng.integers(20, 24, n)).astype(np.float32)
    diag = np.maximum(0, a["ref_start"] - a["query_start"])
    if not shuffle:
        order = (np.lexsort((-a["n_hits"], a["ref_id"], a["is_rc"])) if mate1
                 else np.lexsort((-a["n_hits"], diag, a["ref_id"], a["is_rc"])))
        a = a[order]
    return a


@pytest.mark.gpu
@pytest.mark.parametrize("tries,shuffle,same", [(20, False, False), (20, True, False), (40, False, False),
                                                (3, False, False), (20, False, True)])
def test_long_nam_lists_against_oracle(tries, shuffle, same):
    import torch

    rng = np.random.default_rng(5 + tries + 2 * shuffle + 4 * same)
    ends = []
    for n1 in SIZES:
        for n2 in SIZES:
            if n1 * n2 > 400_000:
                continue
            n_refs, spread = int(rng.choice([1, 1, 3, 12])), int(rng.choice([40, 900, 5000]))
            ends += [make_list(rng, n1, n_refs, spread, True, shuffle), make_list(rng, n2, n_refs, spread, False,
                                                                               shuffle)]
            if same:   # entries the comparator cannot tell apart (it does not look at the reference id)
                for e in ends[-2:]:
                    for f in ("query_start", "query_end", "ref_start", "ref_end", "score"):
                        e[f] = e[f][0] if len(e) else 0
    counts = np.array([len(e) for e in ends])
    nams = np.concatenate(ends)
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
    p = len(ends) // 2
    types = oracle_py.classify_pairs(nams, offs, p, abi.GBSA_PAIRS_INTERLEAVED, 0.5, 300.0, 100.0)
    jp, jc = oracle_py.nam_pairs(nams, offs, p, abi.GBSA_PAIRS_INTERLEAVED, 300.0, 100.0, tries)
    plans, steps = oracle_py.plan_pairs(nams, offs, p, types, jp, jc, max_tries=tries, dropoff=0.3)
    dev = torch.device("cuda:0")
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x).view(np.uint8).copy()).to(dev)
    d_n, d_o, d_t = up(nams), up(offs), up(types)
    d_p = torch.zeros(p * tries * 3, dtype=torch.int32, device=dev)
    d_c = torch.zeros(p, dtype=torch.int32, device=dev)
    native.nam_pairs_device(d_n.data_ptr(), d_o.data_ptr(), p, d_p.data_ptr(), d_c.data_ptr(), 0, 300.0, 100.0, tries)
    torch.cuda.synchronize()
    got_c = d_c.cpu().numpy().astype(np.uint32)
    got_p = d_p.cpu().numpy().view(abi.NAM_PAIR).reshape(p, tries)
    assert (got_c == jc).all()
    for i in range(p):
        assert (got_p[i, : jc[i]] == jp[i, : jc[i]]).all(), (i, counts[2 * i], counts[2 * i + 1])
    cap = len(steps) + 8
    d_plans = torch.zeros(p * abi.PAIR_PLAN.itemsize, dtype=torch.uint8, device=dev)
    d_steps = torch.zeros(cap * abi.ALIGN_STEP.itemsize, dtype=torch.uint8, device=dev)
    n = native.plan_pairs_device(d_n.data_ptr(), d_o.data_ptr(), p, d_t.data_ptr(), d_p.data_ptr(), d_c.data_ptr(),
                                 d_plans.data_ptr(), d_steps.data_ptr(), cap, 0, tries, 0.3)
    torch.cuda.synchronize()
    assert n == len(steps)
    assert (d_plans.cpu().numpy().view(abi.PAIR_PLAN) == plans).all()
    assert (d_steps.cpu().numpy().view(abi.ALIGN_STEP)[:n] == steps).all()
