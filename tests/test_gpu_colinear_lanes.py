"""The colinear sketch and probe with every number of lanes a read may have (1, 2, 4, 8, 16 and 32),
against the oracle: read lengths at the edges of the lanes' stretches."""
import numpy as np
import pytest

import dnaln_b200 as D
from test_gpu_colinear import genome, make_reads
from test_gpu_map import assert_same_as

pytestmark = pytest.mark.gpu


# lanes are doubled while n * lanes stays within the resident ones and the longest read leaves each 32 bases
@pytest.mark.parametrize("n,longest", [(300, 40), (300, 64), (300, 65), (300, 128), (300, 256), (300, 512), (300, 1024),
                                       (300, 1100), (30_000, 150), (60_000, 150)])
def test_every_lane_count_matches_port(ctx, port, n, longest):
    rng = np.random.default_rng(longest)
    g = genome(rng)
    lengths = [longest] + [int(x) for x in rng.integers(1, longest + 1, 60)] + [24, 25, 26, 33, 34, 35]
    base = make_reads(rng, g, min(n, 300), [min(x, longest) for x in lengths])
    seqs = [base.read(i) for i in range(len(base))]
    times = -(-n // len(seqs))
    reads = D.ReadBatch.from_lists(seqs * times, [b"r"] * (len(seqs) * times))
    one = D.ReadBatch.from_lists(seqs, [b"r"] * len(seqs))
    rec, cig, co = port.map(port.index(g), one, D.default_map_params())
    iid = ctx.index_build(g)
    try:
        res = ctx.map_batch(iid, reads)
    finally:
        ctx.index_free(iid)
    off = np.concatenate([co[:-1] + t * co[-1] for t in range(times)] + [[times * co[-1]]])
    assert_same_as((np.tile(rec, (times, 1)), np.tile(cig, times), off), res, len(reads))
