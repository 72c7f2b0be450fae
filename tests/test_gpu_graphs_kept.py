"""An index build leaves the graphs of batches already captured in use."""
import numpy as np
import pytest

import dnaln_b200 as D
from dnaln_b200 import synth

pytestmark = pytest.mark.gpu


def test_an_index_build_keeps_captured_batches():
    with D.Context(0) as c:
        g = synth.make_genome(synth.GenomeSpec(n_contigs=2, contig_len=100_000, gc=0.5), 11)
        big = synth.make_genome(synth.GenomeSpec(n_contigs=2, contig_len=6_000_000, gc=0.5), 12)
        reads, _ = synth.make_reads(g, synth.ReadsSpec(n_reads=500), 13)
        iid = c.index_build(g)
        want = [c.map_batch(iid, reads) for _ in range(3)][-1]
        for genome in (big, g, big):
            before = c.stats()["graph_launches"]
            assert before >= 1
            j = c.index_build(genome)
            got = c.map_batch(iid, reads)
            assert c.stats()["graph_launches"] == before + 1
            assert np.array_equal(got.records, want.records) and np.array_equal(got.cigar, want.cigar)
            c.index_free(j)
