"""Synchronous batches that go in two parts: a refusal writes nothing and is counted as in one
part."""
import ctypes as C

import numpy as np
import pytest
import torch

import dnaln_b200 as D
from dnaln_b200 import synth

pytestmark = pytest.mark.gpu

N, LEN = 250_000, 150  # 37 M bases: above the size from which a batch goes in two parts
MARK = 0x5A


@pytest.fixture(scope="module")
def genome():
    return synth.make_genome(synth.GenomeSpec(n_contigs=2, contig_len=300_000, gc=0.5), 5)


class Batch:
    def __init__(self, genome, seed, pinned=True, longest=LEN):
        reads, _ = synth.make_reads(genome, synth.ReadsSpec(n_reads=N, len_min=LEN, len_max=longest,
                                                            len_dist=2 if longest > LEN else 0), seed)
        assert int(reads.seq_off[-1]) >= N * LEN
        place = (lambda t: t.pin_memory()) if pinned else (lambda t: t)
        ins = [reads.seq, reads.seq_off[:-1], reads.seq_len, reads.name_hash().view(np.int32)]
        self.ins = [place(torch.from_numpy(np.ascontiguousarray(a))) for a in ins]
        self.rec = place(torch.full((N, D.MAP_RECORD_DTYPE.itemsize), MARK, dtype=torch.uint8))
        self.cig = place(torch.full((N * 16,), MARK, dtype=torch.int32))
        self.reads = reads

    def map(self, ctx, iid, cap):
        self.rec.fill_(MARK)
        self.cig.fill_(MARK)
        used, p = C.c_int64(), D.default_map_params()
        rc = ctx._lib.dnaln_gpu_map_batch(ctx.handle, iid, *(a.data_ptr() for a in self.ins), N, C.byref(p),
                                          self.rec.data_ptr(), self.cig.data_ptr(), cap, C.byref(used))
        return rc, used.value, ctx._lib.dnaln_gpu_last_error(ctx.handle)

    def untouched(self):
        return bool((self.rec == MARK).all()) and bool((self.cig == MARK).all())


def test_a_refused_batch_writes_nothing(ctx, genome):
    iid = ctx.index_build(genome)
    b = Batch(genome, 1)
    try:
        ctx.set_sub_batch(N)
        rc, used, _ = b.map(ctx, iid, N * 16)
        assert rc == 0
        want = b.rec.clone(), b.cig.clone()
        whole = [b.map(ctx, iid, cap) for cap in (1000, used - 1)]
        ctx.set_sub_batch(0)
        assert used > N and all(r[0] != 0 for r in whole)
        for cap, expect in zip((1000, used - 1), whole):  # short for the first part, for the second only
            ctx.reset_stats()
            assert b.map(ctx, iid, cap) == expect
            assert b.untouched()
            assert ctx.stats()["reads"] == N  # mapped once
        for cap in (used, N * 16):
            assert b.map(ctx, iid, cap)[:2] == (0, used)
            assert torch.equal(b.rec, want[0]) and torch.equal(b.cig, want[1])
    finally:
        ctx.set_sub_batch(0)
        ctx.index_free(iid)


def test_new_reads_replay_both_parts(ctx, genome):
    iid = ctx.index_build(genome)
    batches = [Batch(genome, 10 + s) for s in range(4)]
    try:
        rose = []
        for b in batches:
            before = ctx.stats()["graph_launches"]
            assert b.map(ctx, iid, N * 16)[0] == 0
            rose.append(ctx.stats()["graph_launches"] - before)
        assert rose[-1] == 2, rose
        ctx.set_option("graphs", 0)
        got = batches[-1].rec.clone(), batches[-1].cig.clone()
        assert batches[-1].map(ctx, iid, N * 16)[0] == 0
        assert torch.equal(batches[-1].rec, got[0]) and torch.equal(batches[-1].cig, got[1])
    finally:
        ctx.set_option("graphs", 1)
        ctx.index_free(iid)


def test_halves_with_gaps_between_their_reads(ctx, genome):
    iid = ctx.index_build(genome)
    b = Batch(genome, 40)
    try:
        assert b.map(ctx, iid, N * 16)[0] == 0
        want = b.rec.clone(), b.cig.clone()
        seq = torch.full((N, LEN + 3), ord("N"), dtype=torch.uint8)
        seq[:, :LEN] = b.ins[0][:N * LEN].view(N, LEN)
        b.ins[0] = seq.flatten().pin_memory()
        b.ins[1] = (torch.arange(N, dtype=torch.int64) * (LEN + 3)).pin_memory()
        assert b.map(ctx, iid, N * 16)[0] == 0
        assert torch.equal(b.rec, want[0]) and torch.equal(b.cig, want[1])
    finally:
        ctx.index_free(iid)


@pytest.mark.parametrize("pinned,longest,parts", [(True, LEN, 2), (True, 256, 2), (True, 260, 1), (False, LEN, 1)])
def test_only_short_page_locked_reads_go_in_two_parts(ctx, genome, pinned, longest, parts):
    iid = ctx.index_build(genome)
    b = Batch(genome, 20, pinned, longest)
    try:
        ctx.set_option("graphs", 0)
        ctx.set_sub_batch(N)
        assert b.map(ctx, iid, N * 16)[0] == 0
        ctx.reset_stats()
        assert b.map(ctx, iid, N * 16)[0] == 0
        one = ctx.stats()["launches"]
        ctx.set_sub_batch(0)
        ctx.reset_stats()
        assert b.map(ctx, iid, N * 16)[0] == 0
        launches = ctx.stats()["launches"]
        assert launches == one if parts == 1 else launches > 1.5 * one
    finally:
        ctx.set_sub_batch(0)
        ctx.set_option("graphs", 1)
        ctx.index_free(iid)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two devices to tell them apart")
def test_the_callers_device_stays_current(genome):
    with D.Context(1) as c:
        iid = c.index_build(genome)
        b = Batch(genome, 30)
        torch.cuda.set_device(0)
        assert b.map(c, iid, N * 16)[0] == 0
        assert torch.cuda.current_device() == 0
