"""Reads whose anchors are checked to form one colinear chain (k_sketch_reads, k_probe_reads)
against the oracle and against the full seeding and chaining kernels (option "colinear" 0):
identical records, and identical minimizer and anchor totals. Read lengths at the edges of
the sketch's blocks, its 16-base chunks and the 32 minimizers of a chunk; batch sizes on
every lanes-per-read split; genomes with tandem repeats, inverted and near copies; reads
with Ns, indels (two close together as well), chimeras and junk."""
import numpy as np
import pytest

import dnaln_b200 as D

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGTN", np.uint8)


def genome(rng):
    parts = []
    core = rng.integers(0, 4, 60_000).astype(np.uint8)
    parts.append(core)
    unit = rng.integers(0, 4, 37).astype(np.uint8)
    parts.append(np.tile(unit, 12))  # a tandem repeat
    parts.append(rng.integers(0, 4, 3_000).astype(np.uint8))
    near = core[10_000:10_700].copy()
    near[rng.random(700) < 0.02] = 0
    parts.append(near)  # a copy within the chaining gap of nothing else
    parts.append((3 - core[20_000:20_600])[::-1])  # an inverted copy
    parts.append(np.repeat(core[30_000:30_300], 1))
    parts.append(core[30_000:30_300])  # a tandem duplication
    parts.append(np.full(40, 4, np.uint8))
    parts.append(rng.integers(0, 4, 20_000).astype(np.uint8))
    g = np.concatenate(parts)
    half = len(g) // 2
    return D.Genome(g, [0, half], [half, len(g) - half])


def make_reads(rng, g, n, lengths):
    codes, seqs = g.codes, []
    for i in range(n):
        L = int(lengths[i % len(lengths)])
        a = int(rng.integers(0, len(codes) - L - 40))
        q = codes[a:a + L + 30].copy()
        flaw = int(rng.integers(10))
        if flaw < 4 and L > 20:  # one indel, or two close together
            for _ in range(1 + (flaw == 0)):
                x, m = int(rng.integers(5, L - 5)), int(rng.integers(1, 6))
                q = np.concatenate([q[:x], q[x + m:]]) if rng.integers(2) else \
                    np.concatenate([q[:x], rng.integers(0, 4, m).astype(np.uint8), q[x:]])
        elif flaw == 4:  # a chimera
            b = int(rng.integers(0, len(codes) - L - 40))
            q[L // 2:] = codes[b:b + len(q) - L // 2]
        elif flaw == 5:
            q[int(rng.integers(len(q)))] = 4
        elif flaw == 6:
            x = int(rng.integers(len(q)))
            q[x:x + 12] = rng.integers(0, 4, len(q[x:x + 12]))
        q = q[:L]
        sub = (rng.random(len(q)) < 0.01) & (q < 4)
        q[sub] = rng.integers(0, 4, int(sub.sum()))
        if rng.integers(2):
            q = np.where(q < 4, 3 - q, 4).astype(np.uint8)[::-1]
        seqs.append(ACGT[q].tobytes())
    return D.ReadBatch.from_lists(seqs, [b"r%d" % i for i in range(n)])


LENGTHS = {
    "short": [1, 14, 15, 23, 24, 25, 26, 33, 34, 35, 44, 63, 64, 65, 100, 150, 151, 255, 256, 257],
    "long": [40, 300, 600, 601, 1000, 1500],
}


@pytest.mark.parametrize("kind,n", [("short", 40), ("short", 2_000), ("short", 120_000), ("long", 24), ("long", 1_200),
                                    ("long", 60_000)])
def test_same_as_the_full_kernels(ctx, kind, n):
    rng = np.random.default_rng(n)
    g = genome(rng)
    reads = make_reads(rng, g, min(n, 4_000), LENGTHS[kind])
    if n > len(reads):  # the same reads again, enough for one lane per read
        times = -(-n // len(reads))
        seqs = [reads.read(i) for i in range(len(reads))] * times
        reads = D.ReadBatch.from_lists(seqs, [b"r%d" % i for i in range(len(seqs))])
    iid = ctx.index_build(g)
    got = []
    try:
        for on in (1, 0):
            ctx.set_option("colinear", on)
            ctx.reset_stats()
            res = ctx.map_batch(iid, reads)
            st = ctx.stats()
            got.append((res, {f: st[f] for f in ("mapped", "candidates", "minimizers", "anchors")}))
    finally:
        ctx.set_option("colinear", 1)
        ctx.index_free(iid)
    (a, sa), (b, sb) = got
    assert sa == sb
    assert np.array_equal(a.cigar, b.cigar)
    for f in a.records.dtype.names:
        assert np.array_equal(a.records[f], b.records[f]), f


@pytest.mark.parametrize("min_score,min_anchors,max_gap,band", [(20, 2, 5000, 16), (16, 1, 5000, 16), (40, 3, 60, 2),
                                                                (20, 2, 100, 0)])
def test_chaining_parameters_match_port(ctx, port, min_score, min_anchors, max_gap, band):
    rng = np.random.default_rng(3)
    g = genome(rng)
    reads = make_reads(rng, g, 1_500, LENGTHS["short"] + LENGTHS["long"])
    p = D.default_map_params()
    p.ch = D.ChainParams(max_gap, band, 50, min_score, min_anchors)
    iid = ctx.index_build(g)
    try:
        res = ctx.map_batch(iid, reads, p)
    finally:
        ctx.index_free(iid)
    rec, cig, co = port.map(port.index(g), reads, p)
    r = res.records
    got = np.stack([r["contig"], r["pos"], r["rev"], r["mapq"], r["score"], r["nm"], r["n_cand"]], 1).astype(np.int64)
    assert np.array_equal(got, rec)
    assert np.array_equal(r["cigar_len"], np.diff(co).astype(np.int32))
    assert np.array_equal(res.cigar, cig)
