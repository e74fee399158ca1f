"""The index build against the oracle where its sort and its segments change shape: entry counts
around the group sizes, groups of repeats' copies larger than a warp sorts (few of them, and most
of the table), contigs that meet in a segment's word, N and tied windows at segment bounds, and
contigs too short for a seed."""
import numpy as np
import pytest

from gpu_index_test_gb300 import native, synth
from oracle import oracle_py

pytestmark = pytest.mark.gpu


def genome_of(contigs):
    seq = np.concatenate([np.frombuffer(c, np.uint8) for c in contigs]) if contigs else np.zeros(0, np.uint8)
    lens = np.array([len(c) for c in contigs], np.uint64)
    offs = np.concatenate([[0], np.cumsum(lens[:-1])]).astype(np.uint64) if contigs else np.zeros(0, np.uint64)
    return synth.Genome(seq.copy(), lens, offs)


def random_bases(rng, n):
    return bytes(rng.choice(np.frombuffer(b"ACGT", np.uint8), n))


def check(contigs, r=150, bits=-1, params=None):
    g = genome_of(contigs)
    p = params or native.params_from_read_length(r)
    idx = native.Index.build(p, g, bits=bits)
    o = oracle_py.Index.build(params or oracle_py.params_from_read_length(r), g, bits=bits)
    rs, st = idx.export()
    assert (rs == o.randstrobes()).all() and (st == o.starts()).all()
    a, b = idx.info(), o.info()
    for f in ("filter_cutoff", "distinct_strobemers", "tot_occur_once", "tot_mid_ab", "tot_high_ab", "size"):
        assert getattr(a, f) == getattr(b, f), f
    return idx


@pytest.mark.parametrize("n", [0, 10, 30, 100, 1500, 60_000, 200_000, 210_000, 1_000_000])
def test_table_sizes(n):
    """From an empty table over a few entries to either side of one and two passes (a syncmer
    every five bases: 41 k entries at 205 kbp)."""
    rng = np.random.default_rng(n)
    check([random_bases(rng, n)])


@pytest.mark.parametrize("copies,unit", [(255, 300), (256, 300), (257, 300), (300, 300), (2047, 120), (2048, 100), (2049, 100), (60, 3000)])
def test_repeats_around_the_group_size(copies, unit):
    """Copies of a unit between random stretches in three contigs: their hashes' groups hold at
    least `copies` entries, whose positions come in the contigs' order and must be merged."""
    rng = np.random.default_rng(copies)
    u = random_bases(rng, unit)
    contigs = []
    for c in range(3):
        parts = []
        for _ in range(copies // 3 + (c < copies % 3)):
            parts += [u, random_bases(rng, int(rng.integers(40, 200)))]
        contigs.append(b"".join(parts))
    check(contigs)


def test_a_table_of_repeats_only():
    rng = np.random.default_rng(1)
    u = random_bases(rng, 500)
    check([u * 300, random_bases(rng, 1000), u * 200, b"ACAC" * 5000, b"A" * 9000])


@pytest.mark.parametrize("r", [50, 150, 300, 400])
def test_segment_bounds(r):
    """N, lower case and tied windows around multiples of the segment, contigs that begin in
    the middle of a word and end within one, and short ones."""
    rng = np.random.default_rng(r)
    contigs = [random_bases(rng, int(n)) for n in (1, 5, 19, 20, 21, 33, 63, 64, 65, 2047, 2048, 2067, 2068, 4095, 4117)]
    for at in (2027, 2028, 2047, 2048, 2049, 2067, 2068, 4096, 6144):
        for what in (b"N", b"NN", b"AAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAAA", b"ACACACACACACACACACACACACACACACAC", b"acgt"):
            s = bytearray(random_bases(rng, 8300))
            s[at: at + len(what)] = what
            contigs.append(bytes(s))
    check(contigs, r=r)


def test_windows_wider_than_the_clean_scan():
    rng = np.random.default_rng(9)
    check([random_bases(rng, 30_000), random_bases(rng, 3000)], params=native.params_make(150, 32, 2, 1, 7, 255, 255))
    check([random_bases(rng, 30_000), random_bases(rng, 3000)], params=native.params_make(150, 9, 9, 1, 7, 255, 80))
