"""The device index build against the oracle, bucket for bucket, at the sizes where its tiles
and words can go wrong: contigs that end around a tile (2,048 window ends) or a word (32
bases), that are shorter than a k-mer or a window, empty, or share bases; N runs that start
and end on word borders and contig ends; a second build in the first one's workspace."""
import numpy as np
import pytest

import dnaln_b200 as D

pytestmark = pytest.mark.gpu


def check(ctx, port, g, k, w):
    idx = port.index(g, k, w)
    iid = ctx.index_build(g, k, w)
    try:
        st = ctx.index_stats(iid)
        got = ctx.index_export(iid)
    finally:
        ctx.index_free(iid)
    want = idx.export()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    counts = want[2]
    assert st["max_count"] == (int(counts.max()) if len(counts) else 0)


@pytest.mark.parametrize("k,w", [(15, 10), (4, 1), (21, 11), (28, 255), (14, 10)])
@pytest.mark.parametrize("lens", [[31], [32], [33], [5, 0, 24, 25, 3000], [2047], [2048], [2049], [2048 * 3 + 14],
                                  [4096 + 15 + 9, 2047 + 24, 70_000]])
def test_edges_match_port(ctx, port, lens, k, w):
    rng = np.random.default_rng(sum(lens) + k)
    n = sum(lens)
    codes = rng.integers(0, 4, n).astype(np.uint8)
    codes[rng.random(n) < 0.002] = 4
    for a in (0, 32, 63, 64, 2016, 2048, 2079):  # N runs on and around word borders
        if a + 2 < n:
            codes[a:a + int(rng.integers(1, 40))] = 4
    codes[max(0, n - 3):] = 4
    off = np.concatenate([[0], np.cumsum(lens)[:-1]])
    check(ctx, port, D.Genome(codes, off, lens), k, w)


def test_contigs_that_share_bases_match_port(ctx, port):
    rng = np.random.default_rng(2)
    codes = rng.integers(0, 4, 9_000).astype(np.uint8)
    codes[4_000:4_064] = 4
    check(ctx, port, D.Genome(codes, [0, 0, 1_000, 3_990], [5_000, 2_100, 8_000, 100]), 15, 10)
