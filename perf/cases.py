"""Performance cases: the calls that programs using this framework make, over the range
of sizes, key widths and options that its workloads cover.

A case is a dict of plain values.  ``kind`` says which call it makes:

* ``host``    -- one read set in host memory through ``Job.run`` with the macro-node table
  copied back to host arrays (the library call behind the ``pkmer`` driver).
* ``graph``   -- FASTA resident in HBM through ``Job.run_device``; the macro-node table
  stays on the device for the next stage.
* ``table``   -- counting alone (``Job.count_device``): the sorted (k-mer, count) table on
  the device and the count histogram, as a k-mer counter is used.
* ``load``    -- macro-nodes from an existing (k-mer, count) table in host memory, as the
  PaK-Graph builder does (``Job.load_table``, ``cutoff``, ``build_macro_nodes``).
* ``wire``    -- initial wiring of a resident macro-node table.
* ``contigs`` -- iterative compaction of a resident macro-node table and the walk to
  contigs, copied to the host (``Job.compact``, ``Job.walk``).
* ``batch``   -- many independent read sets in one ``Batch.run``.
* ``serve``   -- a burst of requests of mixed sizes and k through ``Server``.

Read sets are synthetic: uniform genomes with optional planted repeats, reads of fixed
or ragged length from both strands with substitutions, optional N and lowercase bases,
one header line and one sequence line per read.  Every output is a whole number or raw
bytes, so outputs are compared for equality and there is no ``exact``.  How many rows come
out depends on the reads, so results go to arrays with room to spare whose other rows stay
zero; where the library itself owns the result (``wire``, ``batch``) the seed relabels the
four bases of one read set, which changes every k-mer but no row count.
"""
from __future__ import annotations

import itertools
import math
from ctypes import byref, c_void_p

import numpy as np
import torch

import pakman_plus_gb300 as pk
from pakman_plus_gb300 import capi, synth

_READ_CHUNK = 1 << 18  # reads generated at a time
_CTX = []              # the one Context that a program keeps per device


def _context() -> "pk.Context":
    if not _CTX:
        _CTX.append(pk.Context(0))
    return _CTX[0]


# ------------------------------------------------------------------------- the cases ----
def _case(kind, genome, coverage, read_lo, read_hi, k, err=0.005, repeats="", n_rate=0.0, lower=0.0,
          drop_n=False, sets=1, threshold=0):
    return {"kind": kind, "genome": int(genome), "coverage": int(coverage), "read_lo": int(read_lo),
            "read_hi": int(read_hi), "k": int(k), "err": float(err), "repeats": repeats,
            "n_rate": float(n_rate), "lower": float(lower), "drop_n": bool(drop_n), "sets": int(sets),
            "threshold": int(threshold)}


def listed():
    return [
        # a plasmid-sized read set handed over as host bytes: launches and synchronisations
        dict(_case("host", 2000, 15, 100, 100, 32, err=0.01), name="host_tiny_k32"),
        # the bacterial isolate end to end: pinned host FASTA in, macro-node table out
        dict(_case("host", 4_600_000, 80, 100, 100, 32, repeats="families"), name="host_bacterial_k32"),
        # a small genome with its reads on the device
        dict(_case("graph", 1_000_000, 30, 100, 100, 32, err=0.01), name="graph_1mbp_k32"),
        # the benchmark's read set: 254M windows, repeats, 80x
        dict(_case("graph", 4_600_000, 80, 100, 100, 32, repeats="families"), name="graph_bacterial_k32"),
        # long k-mers (128-bit keys) of a larger genome, windows with N dropped
        dict(_case("graph", 25_000_000, 40, 150, 150, 63, err=0.003, repeats="tandem", n_rate=0.0005,
                   drop_n=True), name="graph_longk_k63"),
        # a k-mer counter's use: ragged trimmed reads with N and soft-masked bases, short k
        dict(_case("table", 8_300_000, 12, 36, 151, 21, n_rate=0.002, lower=0.05), name="table_ragged_k21"),
        # low-complexity reads: a few k-mers hold most windows
        dict(_case("table", 1_000_000, 45, 150, 150, 31, err=0.01, repeats="lowcomplexity"),
             name="table_skewed_k31"),
        # an existing k-mer table turned into a graph
        dict(_case("load", 1_000_000, 30, 100, 100, 31), name="load_1mbp_k31"),
        # initial wiring of the bacterial macro-nodes
        dict(_case("wire", 4_600_000, 40, 100, 100, 32, repeats="families"), name="wire_bacterial_k32"),
        # graph to contigs: compaction to the node threshold and the walk
        dict(_case("contigs", 2_300_000, 60, 100, 100, 32, repeats="families", threshold=50_000),
             name="contigs_2mbp_k32"),
        # a sequencing run's worth of small isolates in one launch
        dict(_case("batch", 300_000, 40, 100, 150, 32, sets=12), name="batch_12_k32"),
        # a burst of requests of all sizes
        dict(_case("serve", 1_500_000, 40, 100, 100, 0, sets=10), name="serve_10_mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "graph", "graph", "graph", "table", "table", "load", "wire", "contigs", "batch",
                       "serve"])
    cov = rng.randint(30, 80)
    lo = rng.randint(80, 160)
    hi = lo if rng.random() < 0.6 else lo + rng.randint(1, 60)
    k = rng.choice([21, 25, 31, 32, 32, 33, 47, 63])
    err = rng.choice([0.003, 0.005, 0.01])
    if kind == "host":
        return _case("host", _log(rng, 1000, 2_000_000), cov, lo, hi, k, err)
    if kind == "graph":
        n_rate = rng.choice([0.0, 0.0, 0.0005])
        return _case("graph", _log(rng, 10_000, 5_000_000), cov, lo, hi, k, err,
                     rng.choice(["", "families", "tandem"]), n_rate, 0.0, n_rate > 0 and rng.random() < 0.7)
    if kind == "table":
        return _case("table", _log(rng, 10_000, 6_000_000), cov, lo, hi, rng.choice([11, 15, 21, 31, 32, 55, 64]),
                     err, rng.choice(["", "", "lowcomplexity"]), rng.choice([0.0, 0.002]), rng.choice([0.0, 0.05]))
    if kind == "load":
        return _case("load", _log(rng, 10_000, 1_500_000), cov, lo, hi, k, err)
    if kind == "wire":
        return _case("wire", _log(rng, 10_000, 4_000_000), cov, lo, hi, k, err, "families")
    if kind == "contigs":
        g = _log(rng, 50_000, 2_500_000)
        return _case("contigs", g, rng.randint(50, 80), lo, hi, rng.choice([31, 32, 33, 63]), 0.005, "families",
                     threshold=max(100, g // rng.randint(20, 100)))
    if kind == "batch":
        return _case("batch", _log(rng, 50_000, 400_000), cov, lo, hi, rng.choice([31, 32, 63]), err,
                     sets=rng.randint(4, 16))
    return _case("serve", _log(rng, 100_000, 2_000_000), cov, 100, 100, 0, err, sets=rng.randint(4, 12))


# ------------------------------------------------------------------------ read sets -----
def _n_reads(case) -> int:
    mean = 0.5 * (case["read_lo"] + case["read_hi"])
    return max(8, int(round(case["coverage"] * case["genome"] / mean)))


def _buckets(case, k) -> int:
    """-t: below the per-strand coverage peak of a k-mer, as a user picks it."""
    mean = 0.5 * (case["read_lo"] + case["read_hi"])
    depth = 0.5 * case["coverage"] * max(0.05, (mean - k + 1) / mean)
    return max(3, min(21, int(0.7 * depth)))


def _genome(rng, case) -> np.ndarray:
    n = max(case["genome"], 4 * case["read_hi"])
    g = rng.integers(0, 4, n, dtype=np.uint8)
    if case["repeats"] == "families":  # 20 families of 3 to 6 copies
        synth.plant_repeat_families(rng, g, 20, min(5000, max(200, n // 200)), 3, 6, 0.5)
    elif case["repeats"] == "tandem":  # 10 % tandem and interspersed repeats of period 2-500
        synth.plant_tandem_and_interspersed(rng, g, 0.10 if n >= 50_000 else 0.0, 2, 500, 0.45)
    elif case["repeats"] == "lowcomplexity":
        # a third of the reads from a homopolymer, a third from a dinucleotide repeat
        span = max(n // 3, case["read_hi"] + 1)
        g[:span] = 0
        g[span:2 * span] = np.resize(np.array([0, 1], np.uint8), g[span:2 * span].size)
    return g


def _fasta(case, seed, relabel=None) -> torch.Tensor:
    """The read set's FASTA bytes on the GPU, made from the seed alone (`relabel`: which of
    the 24 orders of the four bases spells it)."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed * 2 + 1)
    genome = torch.from_numpy(_genome(np.random.Generator(np.random.PCG64(seed)), case)).to(dev)
    lo, hi, n = case["read_lo"], case["read_hi"], _n_reads(case)
    order = next(itertools.islice(itertools.permutations(b"ACGT"), (relabel or 0) % 24, None))
    acgt = torch.tensor(order, dtype=torch.uint8, device=dev)
    col = torch.arange(hi, device=dev)
    parts, first = [], 0
    while first < n:
        digits = len(str(first))
        m = min(n, 10 ** digits, first + _READ_CHUNK) - first
        ln = torch.full((m, 1), lo, device=dev) if lo == hi else \
            torch.randint(lo, hi + 1, (m, 1), device=dev, generator=gen)
        start = (torch.rand((m, 1), device=dev, generator=gen, dtype=torch.float64)
                 * (genome.numel() - ln + 1)).long()
        rev = torch.rand((m, 1), device=dev, generator=gen) < 0.5
        pos = start + torch.where(rev, ln - 1 - col, col)
        codes = genome[pos.clamp_(0, genome.numel() - 1)]
        del pos
        codes = torch.where(rev, 3 - codes, codes)
        wrong = torch.rand((m, hi), device=dev, generator=gen) < case["err"]
        codes = torch.where(wrong, codes + torch.randint(1, 4, (m, hi), device=dev, generator=gen,
                                                         dtype=torch.uint8), codes) & 3
        seq = acgt[codes.int()]
        if case["n_rate"] > 0:
            seq[torch.rand((m, hi), device=dev, generator=gen) < case["n_rate"]] = ord("N")
        if case["lower"] > 0:
            seq = torch.where(torch.rand((m, hi), device=dev, generator=gen) < case["lower"], seq | 0x20, seq)
        rec = torch.empty((m, 3 + digits + hi + 1), dtype=torch.uint8, device=dev)
        rec[:, 0] = ord(">")
        rec[:, 1] = ord("r")
        ids = torch.arange(first, first + m, device=dev)
        for d in range(digits):
            rec[:, 1 + digits - d] = (48 + (ids // 10 ** d) % 10).to(torch.uint8)
        rec[:, 2 + digits] = ord("\n")
        rec[:, 3 + digits:3 + digits + hi] = seq
        rec[:, -1] = ord("\n")
        if lo == hi:
            parts.append(rec.reshape(-1))
        else:
            keep = torch.ones_like(rec, dtype=torch.bool)
            keep[:, 3 + digits:3 + digits + hi] = col < ln
            parts.append(rec[keep])
        first += m
    return torch.cat(parts)


def _pinned(t: torch.Tensor) -> np.ndarray:
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _pinned_zeros(shape, dtype) -> np.ndarray:
    n = int(np.prod(shape)) * np.dtype(dtype).itemsize
    return torch.zeros(n, dtype=torch.uint8, pin_memory=True).numpy().view(dtype).reshape(shape)


def _pinned_nodes(rows: int, k: int):
    """Host arrays for a macro-node table, in pinned memory as the API recommends."""
    keys = _pinned_zeros((rows, 1 if k <= 32 else 2), np.uint64).reshape(-1).view(pk.key_dtype(k))
    return keys, _pinned_zeros((rows, 4), np.uint32), _pinned_zeros((rows, 4), np.uint32)


def _distinct(case) -> float:
    """About how many distinct k-mers a read set has (both strands' genome k-mers, and
    those that substitutions and N bases add)."""
    k, mean = case["k"], 0.5 * (case["read_lo"] + case["read_hi"])
    n = _n_reads(case)
    share = max(0.0, mean - k + 1) / mean
    bad = n * mean * (case["err"] + case["n_rate"]) * k * share
    return min(n * mean * share, 4.0 ** k, 2.0 * case["genome"] + bad)


def _row_room(case) -> int:
    """Rows set aside for a macro-node table (a cutoff near 1 keeps every k-mer)."""
    if _buckets(case, case["k"]) <= 5:
        return int(2.3 * _distinct(case)) + 4096
    return 5 * max(case["genome"], 4 * case["read_hi"]) // 2 + 4096


def _params(case, k=None):
    k = k or case["k"]
    return pk.default_params(k=k, num_buckets=_buckets(case, k), coverage=case["coverage"],
                             read_length=case["read_hi"], drop_n=int(case["drop_n"]))


def _set_cases(case):
    """The independent read sets of a batch or burst: genome sizes spread by a factor of 30
    on a logarithmic scale, in mixed order."""
    n = case["sets"]
    return [dict(case, genome=max(2000, int(case["genome"] * 30.0 ** (-((7 * i) % n) / max(1, n - 1)))),
                 k=case["k"] or (31, 32, 63)[i % 3]) for i in range(n)]


# ----------------------------------------------------------------- device outputs -------
class _View:
    """A job's device buffer as an array; keeps the job alive as long as the array."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _view(owner, ptr, shape, typestr) -> torch.Tensor:
    return torch.as_tensor(_View(owner, ptr, shape, typestr), device="cuda")


def _take(st, name, ptr, rows, words, typestr):
    """The job's rows copied to the program's own tensor, on the job's stream (the job's
    buffers are used again by its next call)."""
    if rows:
        st.out[name][:rows].copy_(_view(st.job, ptr, (rows, words), typestr))
    return st.out[name]


def _take_nodes(st, m):
    keys, suf, pre = c_void_p(), c_void_p(), c_void_p()
    capi.check(capi.lib().pk_macro_nodes_device(st.job.handle, byref(keys), byref(suf), byref(pre)),
               "pk_macro_nodes_device")
    return {"keys": _take(st, "keys", keys.value, m, 1 if st.params.k <= 32 else 2, "<i8"),
            "suffix": _take(st, "suffix", suf.value, m, 4, "<i4"),
            "prefix": _take(st, "prefix", pre.value, m, 4, "<i4")}


def _numbers(s):
    return [s.n_reads, s.n_windows, s.n_unique, s.n_kept, s.n_nodes, s.cutoff]


def _host_nodes(arrays):
    keys, suf, pre = arrays
    return {"keys": keys.view("<i8"), "suffix": suf.view("<i4"), "prefix": pre.view("<i4")}


# ------------------------------------------------------------------ prepare and run -----
class _State:
    """What the program keeps between calls."""


def _contig_arrays(case):
    """Room for the compacted map, the partial contigs and the walk's contigs."""
    n, g = case["threshold"], case["genome"]
    w = 1 if case["k"] <= 32 else 2
    return {"keys": _pinned_zeros((n, w), np.int64), "entry_offsets": _pinned_zeros((n + 1,), np.int64),
            "n_prefixes": _pinned_zeros((n,), np.int32), "entries": _pinned_zeros((12 * n, 8), np.int32),
            "wires": _pinned_zeros((13 * n, 3), np.int32), "ext_bases": _pinned_zeros((16 * g + 65536,), np.uint8),
            "contig_offsets": _pinned_zeros((g // 8 + 4096,), np.int64),
            "contig_bases": _pinned_zeros((8 * g,), np.uint8),
            "walk_offsets": _pinned_zeros((g // 8 + 4096,), np.int64), "walk_bases": _pinned_zeros((16 * g,), np.uint8)}


def prepare(case, seed):
    st = _State()
    st.kind, st.case = case["kind"], case
    if st.kind == "batch":
        st.sets = [(_pinned(_fasta(c, i, relabel=seed)), _params(c)) for i, c in enumerate(_set_cases(case))]
        st.batch = pk.Batch(_context(), branches=6)
        st.out = _pinned_nodes(sum(_row_room(c) for c in _set_cases(case)), case["k"])
        return st
    if st.kind == "serve":
        st.server = pk.Server(_context(), workers=6)
        st.sets = [(_pinned(_fasta(c, seed * 100 + i)), _params(c), _pinned_nodes(_row_room(c), c["k"]))
                   for i, c in enumerate(_set_cases(case))]
        return st
    st.params = _params(case)
    fasta = _fasta(case, 0, relabel=seed) if st.kind == "wire" else _fasta(case, seed)
    torch.cuda.synchronize()
    st.stream = torch.cuda.Stream()
    st.job = pk.Job(_context(), stream=st.stream.cuda_stream)
    rows, words, dev = _row_room(case), 1 if case["k"] <= 32 else 2, torch.device("cuda")
    if st.kind == "host":
        st.fasta = _pinned(fasta)
        st.out = _pinned_nodes(rows, case["k"])
    elif st.kind == "table":
        st.fasta = fasta
        room = int(1.3 * _distinct(case)) + 4096
        st.out = {"keys": torch.zeros((room, words), dtype=torch.int64, device=dev),
                  "counts": torch.zeros((room, 1), dtype=torch.int32, device=dev)}
    elif st.kind in ("graph", "load"):
        if st.kind == "load":
            with pk.Job(_context()) as job:
                job.count_device(fasta.data_ptr(), fasta.numel(), st.params)
                st.keys, st.counts = job.table()
        else:
            st.fasta = fasta
        st.out = {"keys": torch.zeros((rows, words), dtype=torch.int64, device=dev),
                  "suffix": torch.zeros((rows, 4), dtype=torch.int32, device=dev),
                  "prefix": torch.zeros((rows, 4), dtype=torch.int32, device=dev)}
    else:
        st.nodes = st.job.run_device(fasta.data_ptr(), fasta.numel(), st.params).n_nodes
        if st.kind == "contigs":
            st.out = _contig_arrays(case)
    return st


def run(st):
    if st.kind == "batch":
        res = st.batch.run(st.sets)
        tab = st.batch.table(out=st.out)
        out = []
        for r, (_, p) in zip(res, st.sets):
            capi.check(r.status, "batch set")
            mn = st.batch.macro_nodes(r, tab, p.coverage)
            out.append(_host_nodes((mn.keys, mn.suffix_counts, mn.prefix_counts)))
        return {"nodes": out, "numbers": [_numbers(r.summary) for r in res[:2]]}
    if st.kind == "serve":
        tickets = [st.server.submit(f, p, out=o) for f, p, o in st.sets]
        infos = [st.server.wait(t) for t in tickets]
        for t in tickets:
            st.server.release(t)
        return {"nodes": [_host_nodes(o) for _, _, o in st.sets], "numbers": [i.summary.n_nodes for i in infos]}
    with torch.cuda.stream(st.stream):
        return _run_job(st)


def _run_job(st):
    job, lib = st.job, capi.lib()
    if st.kind == "host":
        s = job.run(st.fasta, st.params)
        job.macro_nodes(out=st.out)
        return dict(_host_nodes(st.out), numbers=_numbers(s))
    if st.kind == "graph":
        s = job.run_device(st.fasta.data_ptr(), st.fasta.numel(), st.params)
        return dict(_take_nodes(st, s.n_nodes), numbers=_numbers(s))
    if st.kind == "table":
        job.count_device(st.fasta.data_ptr(), st.fasta.numel(), st.params)
        try:
            cut, hist, kept = job.cutoff(st.params.num_buckets)
        except pk.EmptyAfterCutoff as e:
            cut, hist, kept = e.cutoff, e.hist, e.kept
        rows, windows, reads = job.table_info()
        keys, counts = job.table_device()
        return {"keys": _take(st, "keys", keys, rows, 1 if st.params.k <= 32 else 2, "<i8"),
                "counts": _take(st, "counts", counts, rows, 1, "<i4"),
                "hist": hist.view("<i8"), "numbers": [cut, kept, rows, windows, reads]}
    if st.kind == "load":
        job.load_table(st.keys, st.counts, st.params)
        cut, hist, kept = job.cutoff(st.params.num_buckets)
        m = job.build_macro_nodes(0)
        return dict(_take_nodes(st, m), hist=hist.view("<i8"), numbers=[cut, kept, m])
    if st.kind == "wire":
        rows = c_void_p()
        capi.check(lib.pk_wire_macro_nodes(job.handle, st.case["coverage"]), "pk_wire_macro_nodes")
        capi.check(lib.pk_wiring_device(job.handle, byref(rows)), "pk_wiring_device")
        return _view(job, rows.value, (st.nodes, pk.api.WIRING.itemsize // 4), "<i4")
    # contigs, through the calls a C program makes
    o, p = st.out, {n: a.ctypes.data for n, a in st.out.items()}
    info, walk = capi.PkCompactionInfo(), capi.PkWalkInfo()
    capi.check(lib.pk_compact(job.handle, st.case["threshold"], st.case["coverage"], byref(info)), "pk_compact")
    if info.n_entries > len(o["entries"]) or info.ext_bases > o["ext_bases"].size or             info.n_contigs >= o["contig_offsets"].size or info.contig_bases > o["contig_bases"].size:
        raise RuntimeError("the compacted map does not fit the arrays set aside for it")
    capi.check(lib.pk_copy_compacted(job.handle, p["keys"], p["entry_offsets"], p["n_prefixes"], p["entries"],
                                     p["wires"], p["ext_bases"]), "pk_copy_compacted")
    capi.check(lib.pk_copy_partial_contigs(job.handle, p["contig_offsets"], p["contig_bases"]),
               "pk_copy_partial_contigs")
    capi.check(lib.pk_walk(job.handle, byref(walk)), "pk_walk")
    if walk.n_contigs >= o["walk_offsets"].size or walk.contig_bases > o["walk_bases"].size:
        raise RuntimeError("the contigs do not fit the arrays set aside for them")
    capi.check(lib.pk_copy_walk_contigs(job.handle, p["walk_offsets"], p["walk_bases"]), "pk_copy_walk_contigs")
    return dict(o, numbers=[info.n_nodes, info.n_entries, info.n_contigs, info.rounds, walk.n_contigs])


# ----------------------------------------------------------------------------- work -----
def _work_of_set(case, kind):
    w = 8 if case["k"] <= 32 else 16
    mean = 0.5 * (case["read_lo"] + case["read_hi"])
    n = _n_reads(case)
    fasta = n * (mean + 4 + max(1.0, math.log10(n)))
    windows = n * max(0.0, mean - case["k"] + 1)
    distinct = _distinct(case)
    kept = min(distinct, 2.0 * case["genome"])
    nodes = kept * (w + 32)
    if kind == "table":
        return fasta + distinct * (w + 4), windows
    if kind == "load":
        return distinct * (w + 4) + nodes, distinct
    if kind == "wire":
        return kept * (32 + 168), kept
    if kind == "contigs":
        return nodes + case["threshold"] * 400.0 + kept, kept
    return fasta + nodes, windows


def work(case):
    """Bytes: each input read once and each output written once.  Operations: one insertion
    per window (or one step per row) -- integer work, far below any arithmetic peak."""
    one = [_work_of_set(c, case["kind"]) for c in (_set_cases(case) if case["sets"] > 1 else [case])]
    return {"bytes": sum(b for b, _ in one), "flops": sum(f for _, f in one)}
