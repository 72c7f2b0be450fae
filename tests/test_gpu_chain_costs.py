"""The chaining DP where a gap earns instead of costs: the gap cost int(0.01 k dd + 0.5 log2 dd) is
negative for a k below zero, so a predecessor may add more than k. Many small clusters of anchors,
against the oracle."""
import numpy as np
import pytest

import dnaln_b200 as D
from test_gpu_chain_clusters import clustered_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [-30, -10, -1, 0, 1])
def test_chaining_with_any_k_matches_port(ctx, port, k):
    rng = np.random.default_rng(100 + k)
    cp = (5000, 400, 50, -1000, 1)
    sets = []
    for clusters in (6, 8, 20):
        sr, sq, ss = clustered_set(rng, rng.integers(3, 12, clusters), cp[0], 300)
        sets.append((sr, (sq + rng.integers(0, 300, len(sq))).astype(np.int32), ss))
    got = ctx.chain(sets, k, D.ChainParams(*cp))
    for i, ((sr, sq, ss), ch) in enumerate(got):
        (er, eq, es), ech = port.chain(*sets[i], k, cp)
        assert np.array_equal(sr, er) and np.array_equal(sq, eq) and np.array_equal(ss, es), i
        for key in ech:
            assert np.array_equal(ch[key], ech[key]), (i, key)


def test_cluster_counts_and_sizes_at_the_rules_edges(ctx, port):
    """11, 12 and 13 clusters, the largest of 47 to 49 anchors and about a sixth of all."""
    rng = np.random.default_rng(7)
    cp = (300, 16, 50, 20, 1)
    sets = [clustered_set(rng, [m] * c, cp[0], 10) for c in (11, 12, 13) for m in (1, 4, 20)]
    sets += [clustered_set(rng, [m] + [20] * 13, cp[0], 10) for m in (47, 48, 49, 50, 51, 52, 53, 54)]
    sets += [clustered_set(rng, [m] * 14, cp[0], 10) for m in (47, 48, 49)]
    sets += [clustered_set(rng, [10] + [1] * k, cp[0], 10) for k in (49, 50, 51)]
    got = ctx.chain(sets, 15, D.ChainParams(*cp))
    for i, ((sr, sq, ss), ch) in enumerate(got):
        (er, eq, es), ech = port.chain(*sets[i], 15, cp)
        assert np.array_equal(sr, er) and np.array_equal(sq, eq) and np.array_equal(ss, es), i
        for key in ech:
            assert np.array_equal(ch[key], ech[key]), (i, key)


@pytest.mark.parametrize("k,lookback", [(15, 50), (15, 64), (15, 65), (15, 31), (15, 0), (1024, 50), (1025, 50),
                                        (1_000_000, 50)])
def test_sets_around_256_anchors_match_port(ctx, port, k, lookback):
    """Sets of 0, 1 and about 32, 64 and 256 anchors in one cluster and in some: those chained row by
    row and those in tiles, with packed scores of every size."""
    rng = np.random.default_rng(k + lookback)
    cp = (5000, 16, lookback, 20, 1)
    sets = [tuple(np.zeros(0, t) for t in (np.uint32, np.int32, np.uint32))]
    for n in (1, 2, 11, 12, 13, 31, 32, 33, 34, 63, 64, 65, 97, 128, 255, 256, 257, 300):
        for spread in (2, 30, 200):
            sets.append(clustered_set(rng, [n], cp[0], spread))
            if n > 20:
                sets.append(clustered_set(rng, [n - 12] + [1] * 12, cp[0], spread))
    sets.append(sets[0])
    got = ctx.chain(sets, k, D.ChainParams(*cp))
    for i, ((sr, sq, ss), ch) in enumerate(got):
        (er, eq, es), ech = port.chain(*sets[i], k, cp)
        assert np.array_equal(sr, er) and np.array_equal(sq, eq) and np.array_equal(ss, es), i
        for key in ech:
            assert np.array_equal(ch[key], ech[key]), (i, key)
