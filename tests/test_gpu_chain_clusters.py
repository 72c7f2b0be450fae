"""The chaining DP with a lane per cluster of anchors (chain_dp_clusters) against the oracle:
anchor sets of 5, 6 (the fewest it takes), 7, 32, 33 and 100 clusters, one cluster holding
half of the anchors and one more than half, dense and tied positions, lookbacks below and
above 32 and 64."""
import numpy as np
import pytest

import dnaln_b200 as D

pytestmark = pytest.mark.gpu


def clustered_set(rng, sizes, max_gap, spread):
    """Clusters of the given sizes, each more than max_gap from the next or on the other strand."""
    r, q, s = [], [], []
    at, strand = 1000, 0
    for m in sizes:
        step = rng.integers(0, spread, m)  # 0: anchors of one reference position
        rp = at + np.cumsum(step)
        qp = np.cumsum(np.maximum(step + rng.integers(-3, 4, m), 0)) + int(rng.integers(0, 50))
        off = rng.random(m) < 0.15  # anchors of no chain
        qp[off] = rng.integers(0, 2000, int(off.sum()))
        r.append(rp)
        q.append(qp)
        s.append(np.full(m, strand))
        at = int(rp[-1]) + max_gap + 1 + int(rng.integers(0, 3))
        if rng.random() < 0.3:
            strand, at = 1 - strand, int(rng.integers(1000, at))
    r, q, s = (np.concatenate(x) for x in (r, q, s))
    o = rng.permutation(len(r))
    return r[o].astype(np.uint32), q[o].astype(np.int32), s[o].astype(np.uint32)


@pytest.mark.parametrize("cp", [(5000, 16, 50, 20, 2), (60, 5, 10, 0, 1), (300, 64, 80, 30, 3), (5000, 16, 33, 20, 2)])
def test_clusters_match_port(ctx, port, cp):
    rng = np.random.default_rng(11)
    sets = []
    for clusters in (5, 6, 7, 32, 33, 100):
        for spread in (2, 12, 40):
            sets.append(clustered_set(rng, rng.integers(1, 12, clusters), cp[0], spread))
        sets.append(clustered_set(rng, [3 * (clusters - 1)] + [3] * (clusters - 1), cp[0], 20))  # half of the anchors
        sets.append(clustered_set(rng, [3 * (clusters - 1) + 1] + [3] * (clusters - 1), cp[0], 20))
    sets.append(clustered_set(rng, [100] * 8, cp[0], 10))
    got = ctx.chain(sets, 15, D.ChainParams(*cp))
    for i, ((sr, sq, ss), ch) in enumerate(got):
        (er, eq, es), ech = port.chain(*sets[i], 15, cp)
        assert np.array_equal(sr, er) and np.array_equal(sq, eq) and np.array_equal(ss, es), i
        for key in ech:
            assert np.array_equal(ch[key], ech[key]), (i, key)


@pytest.mark.parametrize("cp", [(5000, 16, 50, 20, 2), (60, 5, 1, 0, 1), (300, 64, 80, 30, 3), (5000, 16, 0, 15, 1),
                                (200, 16, 32, 20, 2), (200, 16, 31, 20, 2)])
def test_long_chains_match_port(ctx, port, cp):
    """One or two clusters of every size around the tiles of 32 rows, with ties and strays."""
    rng = np.random.default_rng(12)
    sets = []
    for n in (1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 255, 256, 257, 700):
        for spread in (1, 3, 25):
            sets.append(clustered_set(rng, [n], cp[0], spread))
            sets.append(clustered_set(rng, [n, n // 2 + 1], cp[0], spread))
    got = ctx.chain(sets, 15, D.ChainParams(*cp))
    for i, ((sr, sq, ss), ch) in enumerate(got):
        (er, eq, es), ech = port.chain(*sets[i], 15, cp)
        assert np.array_equal(sr, er) and np.array_equal(sq, eq) and np.array_equal(ss, es), i
        for key in ech:
            assert np.array_equal(ch[key], ech[key]), (i, key)
