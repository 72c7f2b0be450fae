"""stats.launches against the kernels of this library that a profiler sees, launched one by one and
as graphs."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import dnaln_b200 as D
from dnaln_b200 import synth
from helpers import random_tasks

pytestmark = pytest.mark.gpu


def launched(ctx, call):
    ctx.reset_stats()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    if not names:
        pytest.skip("no kernel trace here (another profiler may hold it)")
    return ctx.stats()["launches"], sum("dnb::" in n for n in names)


@pytest.fixture(scope="module")
def genome():
    return synth.make_genome(synth.GenomeSpec(n_contigs=2, contig_len=400_000, gc=0.5), 3)


@pytest.mark.parametrize("n,lo,hi,bw", [(64, 150, 150, 16), (5000, 150, 150, 16), (5000, 100, 300, 16),
                                        (40_000, 150, 150, 16), (20_000, 50, 1000, 64), (5000, 50, 600, 8),
                                        (3000, 100, 300, 100)])
def test_mapping(ctx, genome, n, lo, hi, bw):
    reads, _ = synth.make_reads(genome, synth.ReadsSpec(n_reads=n, len_min=lo, len_max=hi, len_dist=2 if hi > lo else 0), 4)
    p = D.default_map_params(bw=bw)
    iid = ctx.index_build(genome)
    try:
        for options in ({}, {"colinear": 0}, {"warp_seed_only": 1}, {"ungapped": 0}, {"graphs": 0}, {"length_order": 0}):
            try:
                for o, v in options.items():
                    ctx.set_option(o, v)
                for _ in range(4):  # buffers, forms, and where there are graphs the graph
                    ctx.map_batch(iid, reads, p)
                said, seen = launched(ctx, lambda: ctx.map_batch(iid, reads, p))
                assert said == seen > 0, options
            finally:
                for o, v in options.items():
                    ctx.set_option(o, 1 - v)
    finally:
        ctx.index_free(iid)


@pytest.mark.parametrize("n,bw", [(30, 16), (9000, 16), (13_000, 8), (3000, 21), (2000, 64), (500, 100)])
def test_aligning(ctx, n, bw):
    rng = np.random.default_rng(n)
    qs, ts = random_tasks(rng, min(n, 500), bw, max_len=90)
    times = -(-n // len(qs))
    qs, ts = (qs * times)[:n], (ts * times)[:n]
    sp = D.ScoreParams(2, 4, 4, 2, 1, bw)
    for tb in (True, False):
        for _ in range(3):
            ctx.align(qs, ts, tb, sp)
        said, seen = launched(ctx, lambda: ctx.align(qs, ts, tb, sp))
        assert said == seen > 0, tb
