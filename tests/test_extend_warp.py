"""Seed extension and mate rescue on the GPU against the oracle at the sizes where the warp's
comparisons change shape: read lengths around 8, 32 and 64 bases and past the longest one a warp
compares, reads and windows off 4-byte boundaries, bytes that are no A, C, G or T, NAMs off their
window's diagonal or in the wrong orientation, windows cut by the contig's ends, and scoring
parameters under which a mismatch or a match scores nothing."""
import numpy as np
import pytest

from gpu_index_test_gb300 import abi, native
from oracle import oracle_py

COMP = np.full(256, ord("N"), np.uint8)
for a, b in zip(b"ACGTacgt", b"TGCATGCA"):
    COMP[a] = b
LENGTHS = (21, 24, 31, 32, 33, 40, 63, 64, 65, 96, 127, 128, 129, 150, 191, 192, 193, 255, 256, 257, 300, 400, 511, 512,
           513, 700, 1500)


def sequences(rng, max_len, per_len, k):
    """Contigs, reads cut from them (substituted, some with an indel or odd bytes) and a NAM
    each."""
    lens = np.array([4000, 2500, 9001], np.uint64)
    offs = np.array([1, 4003, 6504], np.uint64)   # off 4-byte boundaries, gaps between
    ref = rng.choice(np.frombuffer(b"ACGT", np.uint8), int(offs[-1] + lens[-1]) + 3)
    odd = rng.choice(len(ref), 60, replace=False)
    ref[odd] = rng.choice(np.frombuffer(b"NnacgtUuRIQ\x01\xff", np.uint8), len(odd))
    reads, roffs, rlens, nams = [], [], [], []
    at = 2
    for length in [x for x in LENGTHS if x <= max_len and x >= k]:
        for _ in range(per_len):
            c = int(rng.integers(3))
            p = int(rng.integers(0, int(lens[c]) - length))
            if rng.random() < 0.15:   # hangs over the contig's start or end
                p = 0 if rng.random() < 0.5 else int(lens[c]) - length
            s = ref[int(offs[c]) + p: int(offs[c]) + p + length].copy()
            subs = rng.random(length) < rng.choice([0.0, 0.01, 0.045, 0.055, 0.2])
            s[subs] = rng.choice(np.frombuffer(b"ACGTN", np.uint8), subs.sum())
            rc = bool(rng.integers(2))
            read = COMP[s[::-1]] if rc else s
            qs = int(rng.integers(0, length - k + 1))
            qe = int(rng.integers(qs + k, length + 1))
            n = np.zeros(1, abi.NAM)
            n["ref_id"], n["is_rc"] = c, rc
            n["query_start"], n["query_end"], n["ref_start"], n["ref_end"] = qs, qe, p + qs, p + qe
            kind = rng.random()
            if kind < 0.15:      # off the diagonal
                n["ref_end"] = min(int(lens[c]), p + qe + int(rng.integers(1, 4)))
            elif kind < 0.3:     # the other orientation's coordinates
                n["is_rc"] = not rc
                n["query_start"], n["query_end"] = length - qe, length - qs
            elif kind < 0.4:     # elsewhere
                d = int(rng.integers(0, int(lens[c]) - (qe - qs)))
                n["ref_start"], n["ref_end"] = d, d + qe - qs
            nams.append(n)
            reads.append(np.concatenate([read, np.zeros(int(rng.integers(0, 4)), np.uint8)]))
            roffs.append(at)
            rlens.append(length)
            at += len(reads[-1])
    seqs = np.concatenate([np.zeros(2, np.uint8)] + reads)
    return ref, offs, lens, seqs, np.array(roffs, np.uint64), np.array(rlens, np.uint32), np.concatenate(nams)


def _device(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).cuda() for a in arrays]


@pytest.mark.gpu
@pytest.mark.parametrize("k,params", [(20, None), (20, (0, 8, 12, 1, 10)), (20, (2, 0, 12, 1, 10)),
                                      (20, (2, 8, 12, 1, -5)), (9, (1, 4, 6, 1, 0)), (32, None)])
def test_extension_at_warp_bounds(k, params):
    import torch

    rng = np.random.default_rng(100 + k)
    ref, offs, lens, seqs, roffs, rlens, nams = sequences(rng, 5000, 24, k)
    ap = None if params is None else abi.align_params(*params)
    own = np.arange(len(nams), dtype=np.uint32)
    want = oracle_py.extend_seeds(ref, offs, lens, seqs, roffs, rlens, nams, own, k,
                                  **({} if ap is None else {"params": ap}))
    d = _device(ref, offs, lens, seqs, roffs, rlens, nams, own)
    out = torch.zeros(len(nams) * abi.SEED_ALIGNMENT.itemsize, dtype=torch.uint8, device="cuda")
    p = [x.data_ptr() for x in d]
    native.extend_seeds_device(p[0], p[1], p[2], len(lens), p[3], p[4], p[5], len(rlens), p[6], p[7], len(nams), k,
                               out.data_ptr(), params=ap)
    got = out.cpu().numpy().view(abi.SEED_ALIGNMENT)
    bad = np.nonzero(got != want)[0]
    assert len(bad) == 0, (bad[:5], rlens[bad[:5]], got[bad[:2]], want[bad[:2]])
    assert 0.1 < want["done"].mean() < 0.95


@pytest.mark.gpu
@pytest.mark.parametrize("k,max_len", [(3, 64), (9, 150), (20, 400), (23, 400), (32, 600)])
@pytest.mark.parametrize("mu,sigma", [(300.0, 100.0), (0.0, 20.0), (2000.0, 10.0)])
def test_mate_rescue_at_warp_bounds(k, max_len, mu, sigma):
    import torch

    rng = np.random.default_rng(200 + k)
    ref, offs, lens, seqs, roffs, rlens, nams = sequences(rng, max_len, 20, k)
    mates = rng.integers(0, len(nams), len(nams)).astype(np.uint32)   # mostly unrelated
    mates[::2] = np.arange(0, len(nams), 2)                           # or the read itself
    nams = nams.copy()
    nams["is_rc"][::4] ^= 1
    sub, step = 2 * k // 3, k // 3
    keep = (rlens[mates].astype(int) - sub + step - 1) // step <= 64
    nams, mates = np.ascontiguousarray(nams[keep]), np.ascontiguousarray(mates[keep])
    want = oracle_py.rescue_mates(ref, offs, lens, seqs, roffs, rlens, nams, mates, k, mu=mu, sigma=sigma)
    d = _device(ref, offs, lens, seqs, roffs, rlens, nams, mates)
    out = torch.zeros(len(nams) * abi.MATE_RESCUE.itemsize, dtype=torch.uint8, device="cuda")
    p = [x.data_ptr() for x in d]
    native.rescue_mates_device(p[0], p[1], p[2], len(lens), p[3], p[4], p[5], len(rlens), p[6], p[7], len(nams), k,
                               out.data_ptr(), mu=mu, sigma=sigma)
    got = out.cpu().numpy().view(abi.MATE_RESCUE)
    bad = np.nonzero(got != want)[0]
    assert len(bad) == 0, (bad[:5], got[bad[:2]], want[bad[:2]])
