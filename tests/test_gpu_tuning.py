"""What a context's first batches may fix for its later ones: the reads-per-block choice is timed on
reads the kernel works on."""
import pytest

import dnaln_b200 as D
from dnaln_b200 import synth

pytestmark = pytest.mark.gpu


def test_reads_per_block_are_timed_on_all_reads():
    g, reads, _ = synth.workload("small-1Mbp-10k-150bp", seed=9, n_reads=40_000)
    with D.Context(0) as c:
        iid = c.index_build(g)
        c.map_batch(iid, reads)
        t = c.seed_tuning()
    assert t["tuned"] == 1 and t["reads"] == len(reads)
    assert min(t["ms_64"], t["ms_128"]) > 0.03  # 40,000 reads; a list passed on unread takes 0.005 ms
