"""What a context's first batches may fix for its later ones: a choice of kernel form made on too
few tasks is made again on a batch that has enough, and the reads-per-block choice is timed on
reads the kernel works on."""
import numpy as np
import pytest

import dnaln_b200 as D
from dnaln_b200 import synth
from helpers import random_tasks

pytestmark = pytest.mark.gpu


def entry(c, W, traceback):
    return next(t for t in c.sw_tuning() if t["W"] == W and t["traceback"] == traceback)


def test_sw_form_of_a_small_batch_is_not_final():
    g = synth.make_genome(synth.GenomeSpec(n_contigs=2, contig_len=400_000, gc=0.5), 21)
    spec = dict(big_del_frac=0.6, big_del_min=3, big_del_max=6)
    small, _ = synth.make_reads(g, synth.ReadsSpec(n_reads=64, **spec), 22)
    large, _ = synth.make_reads(g, synth.ReadsSpec(n_reads=60_000, **spec), 23)
    with D.Context(0) as c:
        iid = c.index_build(g)
        c.map_batch(iid, small)
        assert entry(c, 33, 1)["tasks"] < 4096
        got = [c.map_batch(iid, large) for _ in range(4)]
        t = entry(c, 33, 1)
        assert t["tasks"] >= 4096
        timed = {f: ms for f, ms in enumerate((t["ms_inter"], t["ms_intra"], t["ms_narrow"])) if ms > 0}
        assert t["form"] == min(timed, key=timed.get)
        assert c.stats()["graph_launches"] >= 1  # the last run replays a graph of the final form
        c.map_batch(iid, small)
        assert entry(c, 33, 1) == t  # and stays
    for other in got[1:]:
        assert np.array_equal(got[0].records, other.records) and np.array_equal(got[0].cigar, other.cigar)


def test_sw_form_of_a_small_aligner_call_is_not_final():
    rng = np.random.default_rng(5)
    qs, ts = random_tasks(rng, 700, 16, max_len=60)
    with D.Context(0) as c:
        c.set_option("ungapped", 0)
        c.align(qs[:50], ts[:50], True)
        assert entry(c, 33, 1)["tasks"] == 50
        a = c.align(qs * 30, ts * 30, True)
        b = c.align(qs * 30, ts * 30, True)
        assert entry(c, 33, 1)["tasks"] >= 4096
        assert np.array_equal(a.results, b.results) and np.array_equal(a.cigar, b.cigar)


def test_reads_per_block_are_timed_on_all_reads():
    g, reads, _ = synth.workload("small-1Mbp-10k-150bp", seed=9, n_reads=40_000)
    with D.Context(0) as c:
        iid = c.index_build(g)
        c.map_batch(iid, reads)
        t = c.seed_tuning()
    assert t["tuned"] == 1 and t["reads"] == len(reads)
    assert min(t["ms_64"], t["ms_128"]) > 0.03  # 40,000 reads; a list passed on unread takes 0.005 ms
