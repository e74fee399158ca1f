"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case goes through the public entry points of gpu_index_test_gb300.native: building an
index, seeding reads, mapping read batches (plain, batched and host forms), the reference's
find_nams on query randstrobes, and the first alignment steps on the NAMs found.  Genomes and
reads come from the package's seeded generators, with the shapes the benchmark's
configurations name (C1 uniform, C2 repeat-rich, C3 uneven lengths, C4 human-like).

One reference genome and its index stay in hand for many read batches, as in a program that
maps a sequencing run: they depend on the case alone, and the reads on the seed.  Outputs
go into buffers that the program keeps, sized by the case (zeros past what a pass writes); the
entry points that fill host buffers are called through the C-ABI, as such a program does.
"""
import ctypes
from collections import OrderedDict

import numpy as np
import torch

from gpu_index_test_gb300 import abi, native, synth

# ---- cases ----------------------------------------------------------------------------
#
# kind      the entry point a pass goes through (see run)
# config    genome and read shape; mbp: genome size in Mbp; r: index parameters' read length
# units     single-end reads or pairs per pass; len_min, len_max: read lengths (log-uniform)
# paired    share of units that are pairs


def _map(name, form, config, mbp, units, len_min=150, len_max=150, paired=1.0, r=150):
    return {"name": name, "kind": "map_" + form, "config": config, "mbp": mbp, "units": units, "len_min": len_min,
            "len_max": len_max, "paired": paired, "r": r}


def _steps(name, kind, config, mbp, units, length=150, r=150):
    return {"name": name, "kind": kind, "config": config, "mbp": mbp, "units": units, "len_min": length,
            "len_max": length, "paired": 1.0, "r": r}


def listed():
    return [
        # an interactive or served request: 500 pairs against a resident index, one graph launch
        _map("map 1k batched", "batched", "C2", 100, 500),
        # an ordinary batch of a pipeline that keeps its reads on the device
        _map("map 100k device", "device", "C2", 100, 50_000),
        # the benchmark's batch: a whole chunk of a sequencing run, 1M pairs
        _map("map 2M device", "device", "C2", 100, 1_000_000),
        # reads of uneven length (trimmed, merged, mixed libraries), single-end and paired,
        # mapped as work items; 450-500 bp reads and short ones in one batch
        _map("map ragged batched", "batched", "C3", 5, 200_000, 50, 500, 0.5),
        # a human-like genome (interspersed repeat families) whose index is too large for the
        # fused seeding + lookup kernel
        _map("map human-like device", "device", "C4", 775, 500_000),
        # host buffers in, host records out: 250 bp single-end reads, that profile's index
        _map("map host 250bp", "host", "C2", 20, 100_000, 250, 250, 0.0, 250),
        # a new reference: the index built, then taken to the host (to write or share it)
        {"name": "index 20 Mbp", "kind": "index", "config": "C2", "mbp": 20, "r": 150},
        # the reference's seeding interface: query randstrobes of 100 bp reads, to the host
        {"name": "seed 100bp", "kind": "seed", "config": "C1", "mbp": 5, "units": 50_001, "len_min": 100,
         "len_max": 100, "paired": 0.0, "r": 100},
        # the reference's find_nams on queries that a program already has
        {"name": "find_nams", "kind": "find_nams", "config": "C2", "mbp": 20, "units": 5_000, "len_min": 150,
         "len_max": 150, "paired": 0.0, "r": 150},
        # seed extension of each read's best NAM
        _steps("extend 1M", "extend", "C2", 100, 500_000),
        # mate rescue from each read's best NAM
        _steps("rescue mates 1M", "mates", "C2", 100, 500_000),
        # a batch of pairs through classification, pair scoring, planning and its align steps
        _steps("align pairs 50k", "pairs", "C2", 20, 50_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["map_batched", "map_device", "map_device", "map_host", "index", "seed", "find_nams", "extend",
                       "mates", "pairs"])
    config = rng.choice(["C1", "C2", "C2", "C4"])
    c = {"kind": kind, "config": config, "mbp": _log_int(rng, 2, 60), "r": 150}
    if kind == "index":
        c["r"] = rng.choice([100, 150, 250])
        return c
    r = rng.choice([100, 150, 150, 250])
    length = _log_int(rng, max(50, r - 25), r + 50)
    c.update({"r": r, "len_min": length, "len_max": length, "paired": 1.0})
    if kind in ("map_batched", "map_device", "map_host"):
        c["units"] = _log_int(rng, 200, 400_000 if kind != "map_host" else 150_000)
        c["paired"] = rng.choice([0.0, 0.5, 1.0])
        if rng.random() < 0.4:
            c["len_min"], c["len_max"] = 50, rng.choice([300, 500])
    elif kind == "seed":
        c["units"], c["paired"] = _log_int(rng, 500, 100_000), 0.0
    elif kind == "find_nams":
        c["units"], c["paired"] = _log_int(rng, 100, 10_000), 0.0
    elif kind in ("extend", "mates"):
        c["units"] = _log_int(rng, 500, 400_000)
    else:
        c["units"] = _log_int(rng, 500, 50_000)
    return c


# ---- references and handles that a program keeps --------------------------------------

_references = OrderedDict()   # the last few genomes with their indexes and handles


class _Reference:
    def __init__(self, config, mbp, r):
        self.genome = synth.make_genome(synth.genome_params(config, scale=mbp / _full(config), seed=1))
        self.params = native.params_from_read_length(r)
        self.index = native.Index.build(self.params, self.genome)
        self.handles = {}
        self._device = None

    def device_genome(self):
        if self._device is None:
            g = self.genome
            self._device = (_up(g.seq), _up(g.offsets.astype(np.uint64)), _up(g.lengths.astype(np.uint64)))
        return self._device

    def handle(self, key, make):
        if key not in self.handles:
            self.handles[key] = make()
        return self.handles[key]


def _reference(case):
    key = (case["config"], case["mbp"], case["r"])
    if key in _references:
        _references.move_to_end(key)
    else:
        while len(_references) >= 3:
            _references.popitem(last=False)
        _references[key] = _Reference(*key)
    return _references[key]


def _up(a):
    """A numpy array's bytes on the GPU."""
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()


def _pinned(size, dtype):
    return torch.zeros(size, dtype=dtype).pin_memory()


def _pinned_copy(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).pin_memory()


def _check(code):
    if code != abi.GBSA_OK:
        raise native.GbsaError(code, native.lib().gbsa_last_error().decode())


def _full(config):
    """Mbp of a configuration's genome at full size."""
    return {"C1": 5, "C2": 100, "C3": 5, "C4": 3100}[config]


def _read_params(case, seed):
    c4 = case["config"] == "C4"
    insert = max(350 if c4 else 300, case["len_max"] + 100)
    return synth.ReadParams(seed=1000 + seed, n_units=case["units"], len_min=case["len_min"],
                            len_max=case["len_max"], paired_frac=case["paired"], insert_mean=insert,
                            insert_sd=50 if c4 else 30, sub=(0.005, 0.015) if c4 else (0.01, 0.01))


# ---- prepare --------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "index":
        # a new genome for each seed: this is the input here
        scale = case["mbp"] / _full(case["config"])
        genome = synth.make_genome(synth.genome_params(case["config"], scale=scale, seed=1000 + seed))
        p = native.params_from_read_length(case["r"])
        bp = case["mbp"] * 1_000_000
        bits = native.lib().gbsa_pick_bits(ctypes.byref(p), bp)
        return {"kind": kind, "genome": genome, "params": p, "bits": bits, "entries": np.zeros(bp // 4 * 2, np.int64),
                "starts": np.zeros((1 << bits) + 1, np.int64)}
    if kind == "seed":
        key = (case["config"], case["mbp"], "genome")
        if key not in _references:
            while len(_references) >= 3:
                _references.popitem(last=False)
            scale = case["mbp"] / _full(case["config"])
            _references[key] = synth.make_genome(synth.genome_params(case["config"], scale=scale, seed=1))
        reads = synth.make_reads(_references[key], _read_params(case, seed))
        cap = reads.seq.size * 2 // 3 + 64
        return {"kind": kind, "reads": reads, "params": native.params_from_read_length(case["r"]), "cap": cap,
                "queries": np.zeros(3 * cap, np.int64), "offsets": np.zeros(reads.n + 1, np.int64)}
    ref = _reference(case)
    rp = _read_params(case, seed)
    reads = synth.make_reads(ref.genome, rp)
    n = reads.n
    most = 2 * case["units"]   # reads, whatever share of the units are pairs
    cap = 24 * most + 65536
    if kind == "map_host":
        bases = most * case["len_max"]
        m = ref.handle(("host", most, bases), lambda: native.Mapper(ref.index, max_reads=most, max_bases=bases))
        return {"kind": kind, "mapper": m, "n": n, "cap": cap, "seq": _pinned_copy(reads.seq),
                "off": _pinned_copy(reads.offsets), "len": _pinned_copy(reads.lengths),
                "nams": _pinned(cap * 11, torch.int32), "noff": _pinned(most + 1, torch.int64),
                "frac": _pinned(most, torch.float32), "resc": _pinned(most, torch.uint8)}
    if kind in ("map_device", "map_batched"):
        bases = most * case["len_max"]
        s = {"kind": kind, "n": n, "cap": cap, "seq": _up(reads.seq), "off": _up(reads.offsets),
             "len": _up(reads.lengths), "nams": torch.zeros(cap * 11, dtype=torch.int32, device="cuda"),
             "noff": torch.zeros(most + 1, dtype=torch.int64, device="cuda"),
             "frac": torch.zeros(most, dtype=torch.float32, device="cuda"),
             "resc": torch.zeros(most, dtype=torch.uint8, device="cuda")}
        if kind == "map_device":
            s["mapper"] = ref.handle(("device", most, bases),
                                     lambda: native.Mapper(ref.index, max_reads=most, max_bases=bases))
        else:
            items = synth.read_items(rp)
            s["items"], s["n_items"] = _up(items), len(items) - 1
            s["mapper"] = ref.handle(("batched", most, bases),
                                     lambda: native.Batcher(ref.index, max_reads=most, max_bases=bases))
        return s
    if kind == "find_nams":
        queries, offsets = native.randstrobes_query(ref.params, reads)
        m = ref.handle(("find_nams", n), lambda: native.Mapper(ref.index, max_reads=n))
        return {"kind": kind, "mapper": m, "n": n, "cap": cap, "queries": queries, "offsets": offsets,
                "nams": np.zeros(cap * 11, np.int32), "noff": np.zeros(n + 1, np.int64),
                "frac": np.zeros(n, np.float32)}
    g_seq, g_off, g_len = ref.device_genome()
    s = {"kind": kind, "g": (g_seq.data_ptr(), g_off.data_ptr(), g_len.data_ptr(), len(ref.genome.lengths)),
         "k": ref.params.k, "ref": ref}
    if kind in ("extend", "mates"):
        m = ref.handle(("steps", n), lambda: native.Mapper(ref.index, max_reads=n, max_bases=int(reads.seq.size)))
        nams, offs, _, _ = m.map_reads(reads)
        counts = np.diff(offs.astype(np.int64))
        owners = np.nonzero(counts > 0)[0].astype(np.uint32)
        best = nams[offs[:-1][counts > 0].astype(np.int64)]
        of = owners if kind == "extend" else owners ^ 1   # mates are interleaved
        item = (abi.SEED_ALIGNMENT if kind == "extend" else abi.MATE_RESCUE).itemsize
        s.update({"n": n, "m": len(best), "nams": _up(best), "of": _up(of.astype(np.uint32)), "seq": _up(reads.seq),
                  "off": _up(reads.offsets), "len": _up(reads.lengths),
                  "out": torch.zeros(n * item // 4, dtype=torch.int32, device="cuda")})
        return s
    # pairs: mate 1 and mate 2 mapped in the orders the pair scoring takes (halves layout)
    ends = []
    for e, mode in ((0, abi.GBSA_SORT_REF_MATE1), (1, abi.GBSA_SORT_REF_MATE2)):
        m = ref.handle(("mate", e, n), lambda: native.Mapper(ref.index, abi.map_options(sort_mode=mode),
                                                             max_reads=n // 2, max_bases=int(reads.seq.size)))
        ends.append(m.map_reads(synth.Reads(reads.seq, np.ascontiguousarray(reads.offsets[e::2]),
                                            np.ascontiguousarray(reads.lengths[e::2]))))
    nams = np.concatenate([ends[0][0], ends[1][0]])
    offs = np.concatenate([ends[0][1], ends[1][1][1:] + ends[0][1][-1]])
    p, tries = n // 2, 20
    # steps: a type-4 pair lists up to two per joint NAM pair and two first extensions
    cap = p * (2 + 2 * tries)
    z32 = lambda k: torch.zeros(k, dtype=torch.int32, device="cuda")
    s.update({"p": p, "n": n, "tries": tries, "cap": cap, "nams": _up(nams), "noff": _up(offs.astype(np.uint64)),
              "seq": _up(reads.seq), "off": _up(np.concatenate([reads.offsets[0::2], reads.offsets[1::2]])),
              "len": _up(np.concatenate([reads.lengths[0::2], reads.lengths[1::2]])),
              "types": torch.zeros(p, dtype=torch.uint8, device="cuda"), "joint": z32(p * tries * 3), "jc": z32(p),
              "plans": z32(p * abi.PAIR_PLAN.itemsize // 4), "steps": z32(cap * abi.ALIGN_STEP.itemsize // 4),
              "ext": z32(cap * abi.SEED_ALIGNMENT.itemsize // 4), "mr": z32(cap * abi.MATE_RESCUE.itemsize // 4)})
    return s


# ---- run ------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    lib = native.lib()
    if kind == "index":
        index = native.Index.build(s["params"], s["genome"], bits=s["bits"])
        info = index.info()
        if info.size * 2 > s["entries"].size:
            raise ValueError("more entries than the buffer holds")
        _check(lib.gbsa_index_export(index.h, s["entries"].ctypes.data, s["starts"].ctypes.data))
        return {"entries": s["entries"], "starts": s["starts"], "filter_cutoff": int(info.filter_cutoff)}
    if kind == "seed":
        reads, total = s["reads"], ctypes.c_uint64()
        _check(lib.gbsa_randstrobes_query(ctypes.byref(s["params"]), reads.seq.ctypes.data, reads.offsets.ctypes.data,
                                          reads.lengths.ctypes.data, reads.n, s["queries"].ctypes.data, s["cap"],
                                          s["offsets"].ctypes.data, ctypes.byref(total)))
        return {"queries": s["queries"], "offsets": s["offsets"]}
    if kind == "find_nams":
        _check(lib.gbsa_find_nams(s["mapper"].h, s["queries"].ctypes.data, s["offsets"].ctypes.data, s["n"], 0, 0,
                                  s["nams"].ctypes.data, s["cap"], s["noff"].ctypes.data, s["frac"].ctypes.data))
        return {"nams": s["nams"], "offsets": s["noff"], "frac": s["frac"]}
    if kind == "map_host":
        _check(lib.gbsa_map_reads(s["mapper"].h, s["seq"].data_ptr(), s["off"].data_ptr(), s["len"].data_ptr(),
                                  s["n"], s["nams"].data_ptr(), s["cap"], s["noff"].data_ptr(), s["frac"].data_ptr(),
                                  s["resc"].data_ptr()))
        return {"nams": s["nams"], "offsets": s["noff"], "frac": s["frac"], "rescued": s["resc"]}
    st = torch.cuda.current_stream().cuda_stream
    if kind in ("map_device", "map_batched"):
        more = {"d_items": s["items"].data_ptr(), "n_items": s["n_items"]} if kind == "map_batched" else {}
        s["mapper"].map_reads_device(s["seq"].data_ptr(), s["off"].data_ptr(), s["len"].data_ptr(), s["n"],
                                     s["nams"].data_ptr(), s["cap"], s["noff"].data_ptr(), s["frac"].data_ptr(),
                                     s["resc"].data_ptr(), stream=st, **more)
        return {"nams": s["nams"], "offsets": s["noff"], "frac": s["frac"], "rescued": s["resc"]}
    reads = (s["seq"].data_ptr(), s["off"].data_ptr(), s["len"].data_ptr(), s["n"])
    if kind in ("extend", "mates"):
        call = native.extend_seeds_device if kind == "extend" else native.rescue_mates_device
        call(*s["g"], *reads, s["nams"].data_ptr(), s["of"].data_ptr(), s["m"], s["k"], s["out"].data_ptr(), stream=st)
        return s["out"]
    lists = (s["nams"].data_ptr(), s["noff"].data_ptr())
    native.classify_pairs_device(*lists, s["p"], s["types"].data_ptr(), abi.GBSA_PAIRS_HALVES, stream=st)
    native.nam_pairs_device(*lists, s["p"], s["joint"].data_ptr(), s["jc"].data_ptr(), abi.GBSA_PAIRS_HALVES,
                            max_tries=s["tries"], stream=st)
    k = native.plan_pairs_device(*lists, s["p"], s["types"].data_ptr(), s["joint"].data_ptr(), s["jc"].data_ptr(),
                                 s["plans"].data_ptr(), s["steps"].data_ptr(), s["cap"], abi.GBSA_PAIRS_HALVES,
                                 max_tries=s["tries"], stream=st)
    native.run_align_steps_device(*s["g"], *reads, *lists, s["steps"].data_ptr(), k, s["k"], s["ext"].data_ptr(),
                                  s["mr"].data_ptr(), stream=st)
    return {"types": s["types"], "joint": s["joint"], "joint_counts": s["jc"], "plans": s["plans"],
            "steps": s["steps"], "extensions": s["ext"], "rescues": s["mr"]}


# ---- work -----------------------------------------------------------------------------

def work(case):
    """Bytes each pass has to read or write once: reads and their tables in, records out, and
    the index entries and buckets that the queries name (integer work: no flops)."""
    kind = case["kind"]
    if kind == "index":
        bp = case["mbp"] * 1e6
        entries = bp / 5   # syncmer density: one in k - s + 1 bases
        return {"bytes": bp + 16 * entries + 8 * 2 ** (int(np.log2(entries)) - 1), "flops": 0}
    p = native.params_from_read_length(case["r"])
    lo, hi = case["len_min"], case["len_max"]
    length = lo if lo == hi else (hi - lo) / np.log(hi / lo)   # mean of the log-uniform lengths
    n = case["units"] * (1 + case["paired"])
    queries = 2 * max(0.0, (length - p.k + 1) / (p.k - p.s + 1) - p.w_min)   # of a read, both orientations
    nams = {"C1": 2, "C2": 12, "C3": 4, "C4": 9}[case["config"]]             # of a read, about
    reads_in = length + 12
    per = {
        # a query's bucket bounds and first entry, its filter probe and one hit's entry
        "map_device": reads_in + 64 * queries + 44 * nams + 13,
        "map_batched": reads_in + 64 * queries + 44 * nams + 13,
        "map_host": reads_in + 64 * queries + 44 * nams + 13,
        "seed": reads_in + 24 * queries + 8,
        "find_nams": (24 + 64) * queries + 44 * nams + 12,
        # the read and its reference window; NAM, read index and record
        "extend": 2 * length + 44 + 4 + 36,
        # the mate and the part of its window up to where it is expected; NAM, index, record
        "mates": length + 300 + 44 + 4 + 20,
        # NAM lists; about two steps of a pair with their sequences and records
        "pairs": 44 * nams + 4 * length + 12 * 10 + 2 * (20 + 36 + 20) / 2,
    }[kind]
    return {"bytes": n * per, "flops": 0}


def exact(case, seed):
    # whole-number records throughout; the float fields (a NAM's score, the share of found
    # seeds that are not repetitive) are single roundings of ratios of them
    return None
