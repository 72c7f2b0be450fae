"""An uploaded table that also holds keys no k-mer hashes to (2^32 and above, at k = 15): a lookup
walks past them to the key it wants (src/index.hpp:24-38), in every seeding kernel."""
import numpy as np
import pytest

import dnaln_b200 as D
from dnaln_b200 import synth

pytestmark = pytest.mark.gpu

EMPTY = np.uint64(2**64 - 1)


def with_foreign_keys(keys, offs, cnts):
    """The same keys, each behind a foreign one in its home bucket."""
    full = np.nonzero(keys != EMPTY)[0]
    cap = 16
    while cap < 8 * len(full):
        cap *= 2
    k2, o2, c2 = np.full(cap, EMPTY), np.zeros(cap, np.uint32), np.zeros(cap, np.uint32)

    def put(key, off, cnt):
        i = int(key) & (cap - 1)
        while k2[i] != EMPTY:
            i = (i + 1) & (cap - 1)
        k2[i], o2[i], c2[i] = key, off, cnt
    for x in full:
        put((np.uint64(1) << np.uint64(40)) | keys[x], 0, 0)
    for x in full:
        put(keys[x], offs[x], cnts[x])
    return k2, o2, c2


def test_lookups_walk_past_foreign_keys(ctx):
    g = synth.make_genome(synth.GenomeSpec(n_contigs=2, contig_len=12_000, gc=0.5), 3)
    reads, _ = synth.make_reads(g, synth.ReadsSpec(n_reads=400), 4)
    a = ctx.index_build(g)
    keys, offs, cnts, pos = ctx.index_export(a)
    b = ctx.index_upload(g, *with_foreign_keys(keys, offs, cnts), pos)
    try:
        want = ctx.map_batch(a, reads)
        assert int(want.records["n_cand"].astype(bool).sum()) > 390
        for option, value in ((None, 0), ("colinear", 0), ("warp_seed_only", 1)):
            if option:
                ctx.set_option(option, value)
            try:
                got = ctx.map_batch(b, reads)
            finally:
                if option:
                    ctx.set_option(option, 1 - value)
            assert np.array_equal(got.records, want.records), option
            assert np.array_equal(got.cigar, want.cigar), option
    finally:
        ctx.index_free(a)
        ctx.index_free(b)
