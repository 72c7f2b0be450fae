"""The sums over a batch's reads (packed offsets, seeding totals, CIGAR offsets) at the sizes
where their blocks begin: one block of offsets and several, one group of record blocks and
several, blocks of more than one tile of offsets, and reads that are handed to the warp
kernels directly and through the lists. Every copy of a read gives the record of the read
alone, and the CIGARs lie one behind the other."""
import numpy as np
import pytest

import dnaln_b200 as D

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGTN", np.uint8)


@pytest.fixture(scope="module")
def setup(ctx):
    rng = np.random.default_rng(17)
    unit = rng.integers(0, 4, 700).astype(np.uint8)
    g = np.concatenate([rng.integers(0, 4, 20_000).astype(np.uint8), unit, rng.integers(0, 4, 9_000).astype(np.uint8),
                        unit, rng.integers(0, 4, 5_000).astype(np.uint8)])
    genome = D.Genome(g, [0], [len(g)])
    seqs = []
    for i in range(61):
        L = int(rng.integers(1, 90)) if i else 40
        a = int(rng.integers(0, len(g) - L)) if i % 7 else 20_000 + i  # some from the copies
        q = g[a:a + L].copy()
        if i % 5 == 0 and L > 30:
            q = np.delete(q, [L // 2, L // 2 + 1])
        if i % 11 == 0:
            q[len(q) // 3] = 4
        seqs.append(ACGT[q].tobytes())
    iid = ctx.index_build(genome)
    yield iid, seqs
    ctx.index_free(iid)


def tiled(seqs, n):
    base = D.ReadBatch.from_lists(seqs, [b"x"] * len(seqs))
    times = -(-n // len(seqs))
    off = np.concatenate([[0], np.cumsum(np.tile(base.seq_len.astype(np.int64), times)[:n])])
    return D.ReadBatch(np.tile(base.seq, times)[:off[-1]], off, np.full(n, ord("x"), np.uint8), np.arange(n + 1))


@pytest.mark.parametrize("n", [1, 61, 255, 256, 257, 4095, 4096, 4097, 5121, 16_384, 16_385, 70_001, 2_100_000])
def test_every_copy_of_a_read_gets_its_record(ctx, setup, n):
    iid, seqs = setup
    ctx.reset_stats()
    one = ctx.map_batch(iid, tiled(seqs, len(seqs)))
    s1 = ctx.stats()
    ctx.reset_stats()
    got = ctx.map_batch(iid, tiled(seqs, n))
    st = ctx.stats()
    m = len(seqs)
    r = got.records
    assert len(r) == n
    for f in r.dtype.names:
        if f not in ("cigar_off", "pad_"):
            assert np.array_equal(r[f], np.tile(one.records[f], -(-n // m))[:n]), f
    length = r["cigar_len"].astype(np.int64)
    assert np.array_equal(r["cigar_off"], np.concatenate([[0], np.cumsum(length)[:-1]]))
    copies = n // m
    if copies:
        total = int(one.records["cigar_len"].sum())
        assert np.array_equal(got.cigar[:copies * total], np.tile(one.cigar[:total], copies))
    if n % m == 0:
        for f in ("mapped", "candidates", "minimizers", "anchors", "cells"):
            assert st[f] == s1[f] * copies, f
