"""The sums over a batch's reads (packed offsets, seeding totals, CIGAR offsets) at the sizes
where their blocks begin: one block of offsets and several, one group of record blocks and
several, blocks of more than one tile of offsets, and reads that are handed to the warp
kernels directly and through the lists. Every copy of a read gives the record of the read
alone, and the CIGARs lie one behind the other."""
import ctypes as C
import threading

import numpy as np
import pytest

import dnaln_b200 as D
from dnaln_b200._native import ptr

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


@pytest.mark.parametrize("order", ["packed", "gaps", "shuffled"])
def test_a_large_batch_in_two_parts(ctx, setup, order):
    """16 Mi bases and more go in two parts where the halves' reads lie apart: same results as
    in one part, and a CIGAR buffer that is too small is refused with the same error."""
    iid, seqs = setup
    n = 420_000
    batch = tiled(seqs, n)
    if order != "packed":
        rng = np.random.default_rng(3)
        ln = batch.seq_len.astype(np.int64)
        perm = rng.permutation(n) if order == "shuffled" else np.arange(n)
        place = np.empty(n, np.int64)
        place[perm] = np.concatenate([[0], np.cumsum(ln[perm] + 3)[:-1]])
        seq = np.full(int((ln + 3).sum()), ord("N"), np.uint8)
        at = np.repeat(place - batch.seq_off[:-1], ln) + np.arange(batch.seq_off[-1])
        seq[at] = batch.seq
        batch = (seq, place, batch.seq_len)
    assert int(tiled(seqs, n).seq_off[-1]) >= 16 << 20
    lib, p = ctx._lib, D.default_map_params()
    seq, off, ln = batch if isinstance(batch, tuple) else (batch.seq, batch.seq_off[:-1].copy(), batch.seq_len)
    seq, names = np.ascontiguousarray(seq), np.full(n, 7, np.uint32)

    def run(cap):
        rec, cig, used = np.zeros(n, D.MAP_RECORD_DTYPE), np.zeros(cap, np.uint32), C.c_int64()
        rc = lib.dnaln_gpu_map_batch(ctx.handle, iid, ptr(seq), ptr(off), ptr(ln), ptr(names), n, C.byref(p), ptr(rec),
                                     ptr(cig), cap, C.byref(used))
        return rc, rec, cig[:used.value], used.value, lib.dnaln_gpu_last_error(ctx.handle)

    try:
        ctx.set_sub_batch(n)
        want, small = run(8 * n), run(1000)
        ctx.set_sub_batch(0)
        got, refused = run(8 * n), run(1000)
    finally:
        ctx.set_sub_batch(0)
    assert got[0] == want[0] == 0 and got[3] == want[3]
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    assert refused[0] == small[0] != 0 and refused[3] == small[3] and refused[4] == small[4]


def test_calls_from_threads_and_queued_batches(ctx, setup):
    """Batches mapped in the calling thread while others are queued and mapped by other threads."""
    iid, seqs = setup
    batches = [tiled(seqs, n) for n in (61, 700, 5_000, 20_000)]
    want = [ctx.map_batch(iid, b) for b in batches]
    bad = []

    def work(k):
        for i in range(12):
            x = (i + k) % len(batches)
            if (i + k) % 3 == 0:
                got = ctx.map_wait(ctx.map_submit(iid, batches[x]))
            else:
                got = ctx.map_batch(iid, batches[x])
            if not (np.array_equal(got.records, want[x].records) and np.array_equal(got.cigar, want[x].cigar)):
                bad.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
