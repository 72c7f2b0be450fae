"""The mapping path's performance cases: what a user of this framework has it do, through
the C ABI (include/dnaln_b200.h) and its Python mirror.

Three kinds of work:

* ``map``   one batch of reads against a resident index (Mapper::map), either from host
            buffers (``where = "host"``: page-locked arrays in, records and CIGARs out,
            dnaln_gpu_map_batch) or with every buffer on the device (``where = "device"``,
            dnaln_gpu_map_batch_device);
* ``align`` a batch of banded Smith-Waterman tasks from host buffers (Aligner::align,
            dnaln_gpu_align), score only or with traceback;
* ``open``  a genome made resident (dnaln_gpu_index_build) and its first reads mapped, as
            every mapping process starts.

A program keeps one context and its resident index and maps batch after batch, so the
context and the index of a case are made once and kept while the case is in use; a state
is one batch of reads (or tasks) of its own seed, with the buffers of its results. Reads
follow the workloads of ``dnaln_b200.synth``: 1% substitutions, 0.1% indels, and, where a
case says so, long deletions. Every output is a whole number (records, CIGAR operations,
alignment results), compared bit for bit.
"""
import ctypes as C
import functools
import json

import numpy as np
import torch

import dnaln_b200 as D
from dnaln_b200 import synth

RECORD_BYTES = D.MAP_RECORD_DTYPE.itemsize
RESULT_BYTES = D.ALIGN_RESULT_DTYPE.itemsize


def _map(name, where, genome_bp, n, len_min, len_max, dist="uniform", bw=16, repeats=False, big_del=0.0):
    return {"name": name, "kind": "map", "where": where, "genome_bp": genome_bp, "repeats": repeats, "n": n,
            "len_min": len_min, "len_max": len_max, "dist": dist, "big_del": big_del, "bw": bw}


def _align(name, n, len_min, len_max, bw, traceback):
    return {"name": name, "kind": "align", "genome_bp": 4_600_000, "repeats": False, "n": n, "len_min": len_min,
            "len_max": len_max, "dist": "uniform", "big_del": 0.0, "bw": bw, "traceback": traceback}


def _open(name, genome_bp, n):
    return {"name": name, "kind": "open", "genome_bp": genome_bp, "repeats": False, "n": n, "len_min": 150,
            "len_max": 150, "dist": "uniform", "big_del": 0.0, "bw": 16}


def listed():
    return [
        # an interactive request: a handful of reads, where the call's latency is all there is
        _map("request-64", "host", 4_600_000, 64, 100, 300),
        # the request server's mean request
        _map("request-4557", "host", 4_600_000, 4_557, 100, 300),
        # the small whole job: 10,000 reads on a 1 Mbp genome
        _map("small-10k", "host", 1_000_000, 10_000, 150, 150),
        # the headline workload's batch (1,000,000 x 150 bp run as batches of this size), resident in HBM
        _map("batch-150", "device", 4_600_000, 262_144, 150, 150),
        # the same batch from the host's buffers in one synchronous call, copies included
        _map("stream-150", "host", 4_600_000, 262_144, 150, 150),
        # reads of uneven length with long deletions, a ragged count, the default band
        _map("mixed-bw16", "device", 4_600_000, 200_003, 50, 1000, "log", 16, big_del=0.02),
        # the same kind at the widest band in use
        _map("mixed-bw64", "device", 4_600_000, 100_003, 50, 1000, "log", 64, big_del=0.02),
        # a repeat-rich genome of eight contigs with N runs: many candidates per read
        _map("repeat-150", "device", 120_000_000, 262_144, 150, 150, repeats=True),
        # long reads, past what the thread-per-read kernels hold
        _map("long-bw32", "device", 4_600_000, 4_001, 1000, 5000, "uniform", 32),
        # the aligner alone, as a mapper that keeps its own seeding calls it: with traceback
        _align("align-tb", 50_001, 50, 400, 16, True),
        # and score only, as candidates are ranked, at the widest band
        _align("align-score-bw64", 50_001, 100, 300, 64, False),
        # a process's start: the index built on the device, the first reads mapped
        _open("open-4.6M", 4_600_000, 4_096),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["map", "map", "map", "map", "map", "map", "align", "align", "open"])
    if kind == "open":
        return {k: v for k, v in _open("", _log_int(rng, 500_000, 4_600_000), _log_int(rng, 64, 4_096)).items()
                if k != "name"}
    bw = rng.choice([8, 16, 16, 16, 21, 32, 64])
    shape = rng.choice(["fixed", "uniform", "log", "long"] if kind == "map" else ["fixed", "uniform", "log"])
    big_del = 0.0
    if shape == "fixed":
        a = b = rng.randint(50, 256)
    elif shape == "uniform":
        a = rng.randint(40, 200)
        b = a + rng.randint(1, 200)
    elif shape == "log":
        a, b, big_del = rng.randint(40, 100), rng.randint(400, 1000), rng.choice([0.0, 0.02])
    else:
        a = rng.randint(600, 2000)
        b = a + rng.randint(1, 3000)
    # at most the cells and bases of the largest listed case of the kind
    cells = 250_000_000 if shape == "long" else (2_000_000_000 if kind == "map" else 400_000_000)
    n_max = int(min(262_144 if kind == "map" else 50_001, cells // ((a + b) / 2 * (2 * bw + 1)),
                    39_000_000 // ((a + b) / 2), 2_000 if shape == "long" else 262_144))
    n = _log_int(rng, 64, max(n_max, 65))
    if kind == "align":
        c = _align("", n, a, b, bw, rng.random() < 0.6)
        c["dist"] = "log" if shape == "log" else "uniform"
    else:
        bp, repeats = rng.choice([(1_000_000, False), (4_600_000, False), (2_000_000, True), (24_000_000, True)])
        c = _map("", rng.choice(["host", "device"]), bp, n, a, b, "log" if shape == "log" else "uniform", bw, repeats,
                 big_del)
    del c["name"]
    return c


# ---- what a program keeps: a context, a genome, its resident index ------------------------
@functools.lru_cache(maxsize=4)
def _genome(genome_bp, repeats):
    if repeats:
        # the 120 Mbp workload's composition, repeat density and N runs, at any size
        spec = synth.GenomeSpec(n_contigs=8, contig_len=genome_bp // 8, gc=0.42,
                                n_repeat_units=max(8, genome_bp // 600_000), repeat_unit_len=2000, repeat_frac=0.06,
                                repeat_div=0.02, n_frac=0.005, n_run_min=10, n_run_max=100)
    else:
        spec = synth.GenomeSpec(contig_len=genome_bp)
    return synth.make_genome(spec, 11)


class _Program:
    """One context with the case's index resident, and the parameters of its calls."""

    def __init__(self, case):
        self.genome = _genome(case["genome_bp"], case["repeats"])
        self.ctx = D.Context(0)
        self.params = D.default_map_params(bw=case["bw"])
        self.index = self.ctx.index_build(self.genome) if case["kind"] == "map" else None


@functools.lru_cache(maxsize=1)
def _program(key):
    return _Program(json.loads(key))


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory()


def _cigar_cap(case):
    """Room for the batch's CIGAR operations, several times what 0.1% of indels ask for."""
    return case["n"] * (16 + case["len_max"] // 16)


def _reads(case, genome, seed):
    dist = {"log": 1, "uniform": 2}[case["dist"]] if case["len_max"] > case["len_min"] else 0
    spec = synth.ReadsSpec(n_reads=case["n"], len_min=case["len_min"], len_max=case["len_max"], len_dist=dist,
                           big_del_frac=case["big_del"], big_del_min=8, big_del_max=15)
    return synth.make_reads(genome, spec, seed)


def prepare(case, seed):
    pr = _program(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True))
    s = {"case": case, "program": pr, "used": C.c_int64(), "lib": D.lib()}
    reads, truth = _reads(case, pr.genome, 1_000 + seed)
    if case["kind"] == "align":
        _tasks(s, case, pr.genome, reads, truth)
        return s
    lens = reads.seq_len
    ins = [reads.seq, reads.seq_off[:-1], lens, reads.name_hash().view(np.int32)]
    s["cap"] = _cigar_cap(case)
    if case["kind"] == "map" and case["where"] == "device":
        s["ins"] = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in ins]
        s["rec"] = torch.zeros(case["n"], RECORD_BYTES, dtype=torch.uint8, device="cuda")
        s["cig"] = torch.zeros(s["cap"], dtype=torch.int32, device="cuda")
    else:
        s["ins"] = [_pinned(a) for a in ins]
        s["rec"] = torch.zeros(case["n"], RECORD_BYTES, dtype=torch.uint8).pin_memory()
        s["cig"] = torch.zeros(s["cap"], dtype=torch.int32).pin_memory()
    if case["kind"] == "open":
        g = pr.genome
        s["genome"] = [_pinned(g.codes), _pinned(g.contig_off.view(np.int64)), _pinned(g.contig_len.view(np.int32))]
    return s


def _tasks(s, case, genome, reads, truth):
    """Each read, in the strand it maps in, against the genome window its candidate gives."""
    n, lens, off = case["n"], reads.seq_len.astype(np.int64), reads.seq_off[:-1]
    table = np.full(256, 4, np.uint8)
    table[np.frombuffer(b"ACGT", np.uint8)] = np.arange(4, dtype=np.uint8)
    codes = table[reads.seq]
    owner = np.repeat(np.arange(n), lens)
    at = np.arange(len(codes)) - off[owner]
    rev = truth.rev.astype(bool)[owner]
    src = off[owner] + np.where(rev, lens[owner] - 1 - at, at)
    q = codes[src]
    q = np.where(rev & (q < 4), 3 - q, q).astype(np.uint8)
    t_off = np.maximum(truth.start - case["bw"], 0)
    t_len = np.minimum(truth.start + lens + case["bw"], len(genome.codes)) - t_off
    cap = _cigar_cap(case) if case["traceback"] else 1
    s["ins"] = [_pinned(a) for a in (q, off, lens.astype(np.int32), genome.codes, t_off, t_len.astype(np.int32))]
    s["rec"] = torch.zeros(n, RESULT_BYTES, dtype=torch.uint8).pin_memory()
    s["cig"] = torch.zeros(cap, dtype=torch.int32).pin_memory()
    s["cap"] = cap if case["traceback"] else 0


def _check(ctx, rc):
    if rc != 0:
        raise D.DnalnError(rc, D.lib().dnaln_gpu_last_error(ctx.handle).decode())


def run(s):
    case, pr, lib, used = s["case"], s["program"], s["lib"], s["used"]
    ctx, p = pr.ctx, [t.data_ptr() for t in s["ins"]]
    if case["kind"] == "align":
        q, qo, ql, t, to, tl = p
        _check(ctx, lib.dnaln_gpu_align(ctx.handle, q, qo, ql, t, to, tl, case["n"], int(case["traceback"]),
                                        C.byref(pr.params.sc), s["rec"].data_ptr(), s["cig"].data_ptr(), s["cap"],
                                        C.byref(used)))
        return {"results": s["rec"], "cigar": s["cig"], "used": used.value}
    seq, off, lens, names = p
    index = pr.index
    stats = None
    if case["kind"] == "open":
        iid, codes, co, cl = C.c_int32(), *[t.data_ptr() for t in s["genome"]]
        _check(ctx, lib.dnaln_gpu_index_build(ctx.handle, codes, len(pr.genome.codes), co, cl, pr.genome.n_contigs,
                                              pr.params.k, pr.params.w, C.byref(iid)))
        index = iid.value
        stats = ctx.index_stats(index)
    call = lib.dnaln_gpu_map_batch_device if case.get("where") == "device" else lib.dnaln_gpu_map_batch
    _check(ctx, call(ctx.handle, index, seq, off, lens, names, case["n"], C.byref(pr.params), s["rec"].data_ptr(),
                     s["cig"].data_ptr(), s["cap"], C.byref(used)))
    out = {"records": s["rec"], "cigar": s["cig"], "used": used.value}
    if stats is not None:
        ctx.index_free(index)
        out["index"] = np.array([stats[k] for k in ("n_keys", "n_positions", "max_count", "n_buckets")], np.int64)
    return out


def _mean_len(case):
    a, b = case["len_min"], case["len_max"]
    return (b - a) / np.log(b / a) if case["dist"] == "log" and b > a else (a + b) / 2


def work(case):
    """Bytes of one pass. The path's arithmetic is integer throughout, so no floating-point operations."""
    n, length = case["n"], _mean_len(case)
    window = length + 2 * case["bw"]  # target bases of an alignment, one code byte each
    if case["kind"] == "align":
        ops = 3 * 4 if case["traceback"] else 0
        return {"bytes": n * (length + min(window, case["genome_bp"]) + 24 + RESULT_BYTES + ops), "flops": 0.0}
    # a read's bases and its offset, length and name hash in; its record and a few CIGAR operations out;
    # its window of the genome; a 32-byte sector of the table and one of the positions per minimizer
    per_read = length + 16 + RECORD_BYTES + 12 + window + 2 * 32 * length * 2 / 11
    total = n * per_read
    if case["kind"] == "open":
        # the genome's codes in; the buckets (16 bytes, at most half of them full) and the positions written
        minimizers = case["genome_bp"] * 2 / 11
        total += case["genome_bp"] + 2 * 16 * minimizers + 4 * minimizers
    return {"bytes": float(total), "flops": 0.0}


def exact(case, seed):
    """Whole numbers only: they are equal or wrong, so there is no 64-bit value to be near to."""
    return None
