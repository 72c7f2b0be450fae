"""Reads of 257 to 1,024 anchors, which k_chain_map lists for k_chain_big, and reads on either
side of that range, against the oracle: a genome with nine copies of one unit, some of them cut short,
and reads of every length that brings the anchor counts to the edges."""
import numpy as np
import pytest

import dnaln_b200 as D

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGTN", np.uint8)
EDGES = (256, 257, 1024, 1025)


@pytest.fixture(scope="module")
def copies():
    rng = np.random.default_rng(5)
    unit = rng.integers(0, 4, 1_500).astype(np.uint8)
    parts = [rng.integers(0, 4, 9_000).astype(np.uint8)]
    for c in range(9):
        u = unit[:1_500 - 90 * c].copy()
        parts += [3 - u[::-1] if c % 3 == 1 else u, rng.integers(0, 4, 6_000).astype(np.uint8)]
    g = np.concatenate(parts)
    return D.Genome(g, [0], [len(g)]), unit


@pytest.mark.parametrize("stealing", [0, 1])
def test_reads_with_many_anchors_match_port(ctx, port, copies, stealing):
    g, unit = copies
    rng = np.random.default_rng(6)
    seqs = []
    for L in list(range(60, 260, 2)) + list(range(260, 1_500, 5)) + [1_500] * 3:
        q = unit[:L].copy()
        if L % 3 == 0:
            sub = rng.random(L) < 0.02
            q[sub] = rng.integers(0, 4, int(sub.sum()))
        if L % 20 == 0:
            q[L // 2] = 4
        seqs.append(ACGT[q].tobytes())
    reads = D.ReadBatch.from_lists(seqs, [b"r%d" % i for i in range(len(seqs))])
    iid = ctx.index_build(g)
    try:
        ctx.set_option("work_stealing", stealing)
        counts = []
        for s in seqs[::7]:  # the ranges below, between and above the edges are all met
            ctx.reset_stats()
            ctx.map_batch(iid, D.ReadBatch.from_lists([s], [b"x"]))
            counts.append(ctx.stats()["anchors"])
        assert min(counts) < EDGES[0] and max(counts) > EDGES[-1]
        assert any(EDGES[1] <= c <= EDGES[2] for c in counts)
        res = ctx.map_batch(iid, reads)
    finally:
        ctx.set_option("work_stealing", 1)
        ctx.index_free(iid)
    p = D.default_map_params()
    rec, cig, co = port.map(port.index(g), reads, p)
    r = res.records
    got = np.stack([r["contig"], r["pos"], r["rev"], r["mapq"], r["score"], r["nm"], r["n_cand"]], 1).astype(np.int64)
    assert np.array_equal(got, rec)
    assert np.array_equal(r["cigar_len"], np.diff(co).astype(np.int32))
    assert np.array_equal(res.cigar, cig)
