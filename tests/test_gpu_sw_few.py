"""The banded SW form of four cells per lane (short task lists) and the eight-lane traceback
walk against the oracle, bit for bit, at the sizes where they can go wrong: task counts
around a warp's and a block's pairs, query lengths around the walk's 8- and 64-row blocks,
and a list length read on the device on both sides of the form's limit."""
import numpy as np
import pytest

import dnaln_b200 as D
from helpers import mutate, random_codes, random_tasks
from test_gpu_align import check_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bw", [8, 16, 32, 64])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 31, 33, 400])
def test_four_cells_per_lane_matches_port(ctx, port, bw, n):
    rng = np.random.default_rng(100 * bw + n)
    qs, ts = random_tasks(rng, n, bw)
    sc = (2, 4, 4, 2, 1, bw)
    try:
        ctx.set_option("sw_form", 4)
        for tb in (True, False):
            check_same(ctx.align(qs, ts, tb, D.ScoreParams(*sc)), port.align(qs, ts, tb, sc), tb)
    finally:
        ctx.set_option("sw_form", 0)


@pytest.mark.parametrize("scheme", [(2, 4, 4, 2, 1, 16), (2, 8, 12, 2, 1, 5), (3, 2, 0, 3, 1, 21), (2, 0, 4, 2, 0, 8)])
def test_walk_blocks_match_port(ctx, port, scheme):
    """Diagonal runs that end, by a gap, a clip or the score, at every offset of a 64-row stride."""
    rng = np.random.default_rng(31 + scheme[1])
    bw = scheme[5]
    qs, ts = [], []
    for i in range(420):
        core = random_codes(rng, 60 + i, 0.01 if i % 3 == 0 else 0.0)
        m = np.where(core > 3, 0, core).astype(np.uint8)
        cut = 8 + i % 72
        q = np.concatenate([random_codes(rng, i % 9), core[:cut], random_codes(rng, i % 4), core[cut:]])
        m = mutate(rng, m, 0.004, 0.0)
        shift = int(rng.integers(2 * bw + 1))
        t = np.concatenate([random_codes(rng, shift), m, random_codes(rng, 2 * bw + 16)])
        qs.append(q)
        ts.append(t.astype(np.uint8))
    check_same(ctx.align(qs, ts, True, D.ScoreParams(*scheme)), port.align(qs, ts, True, scheme), True)


@pytest.mark.parametrize("n", [3072, 3073, 3200])
def test_list_length_around_the_forms_limit(ctx, port, n):
    bw = 64  # the smallest limit
    rng = np.random.default_rng(n)
    qs, ts = random_tasks(rng, n, bw, max_len=90)
    sc = (2, 4, 4, 2, 1, bw)
    check_same(ctx.align(qs, ts, True, D.ScoreParams(*sc)), port.align(qs, ts, True, sc), True)
