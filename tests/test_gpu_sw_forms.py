"""Every form of the banded SW kernels against the oracle, bit for bit, where their row loops
and their work lists can go wrong: queries of 1 to 70 rows (shorter than, as long as and just
longer than the skew and the blocks of codes that the lanes of a pair load together), pairs of
very different lengths, and lists longer than the resident warps take at once."""
import numpy as np
import pytest

import dnaln_b200 as D
from helpers import mutate, random_codes, random_tasks
from test_gpu_align import check_same

pytestmark = pytest.mark.gpu


def short_tasks(rng, lengths, bw):
    qs, ts = [], []
    for L in lengths:
        core = np.minimum(random_codes(rng, L + 2 * bw + 8, 0.0), 3)
        s = int(rng.integers(0, 2 * bw + 1))
        q = mutate(rng, core[s:s + L], 0.03, 0.01)[:L]
        qs.append((q if len(q) else core[:1]).astype(np.uint8))
        ts.append(core.astype(np.uint8))
    return qs, ts


@pytest.mark.parametrize("form", [1, 2, 3, 4])
@pytest.mark.parametrize("scheme", [(2, 4, 4, 2, 1, 8), (2, 4, 4, 2, 1, 16), (3, 5, 0, 1, 2, 32), (2, 0, 6, 0, 0, 64)])
def test_row_edges_match_port(ctx, port, form, scheme):
    bw = scheme[5]
    rng = np.random.default_rng(7 * form + bw)
    lengths = list(range(1, 71)) + [1, 70, 64, 2, 300, 1, 33, 500]
    qs, ts = short_tasks(rng, lengths, bw)
    try:
        ctx.set_option("ungapped", 0)
        ctx.set_option("sw_form", form)
        for tb in (True, False):
            check_same(ctx.align(qs, ts, tb, D.ScoreParams(*scheme)), port.align(qs, ts, tb, scheme), tb)
    finally:
        ctx.set_option("sw_form", 0)
        ctx.set_option("ungapped", 1)


@pytest.mark.parametrize("form,bw,n", [(1, 16, 120_000), (2, 64, 24_000), (3, 16, 60_000), (4, 32, 16_000)])
def test_more_pairs_than_resident_warps(ctx, port, form, bw, n):
    """The first 700 tasks again and again: every copy gives the oracle's results."""
    rng = np.random.default_rng(n)
    sc = (2, 4, 4, 2, 1, bw)
    qs, ts = short_tasks(rng, rng.integers(1, 60, 700), bw)
    ra, rb = random_tasks(rng, 50, bw, max_len=60)
    qs, ts = qs[:650] + ra, ts[:650] + rb
    times = -(-n // len(qs))
    want = port.align(qs, ts, True, sc)
    try:
        ctx.set_option("ungapped", 0)
        ctx.set_option("sw_form", form)
        check_same(ctx.align(qs * times, ts * times, True, D.ScoreParams(*sc)), want * times, True)
    finally:
        ctx.set_option("sw_form", 0)
        ctx.set_option("ungapped", 1)


@pytest.mark.parametrize("form", [1, 3, 4])
@pytest.mark.parametrize("scheme", [(2, 4, 4, 2, 1, 5), (2, 4, 4, 2, 1, 21), (3, 2, 0, 3, 1, 21), (2, 0, 4, 2, 0, 5)])
def test_bands_that_end_inside_a_lane(ctx, port, form, scheme):
    """W = 11 and 43 end in the middle of a lane's cells, with idle lanes after it."""
    bw = scheme[5]
    rng = np.random.default_rng(9 * form + bw)
    qs, ts = short_tasks(rng, list(range(1, 71)) + [1, 70, 64, 2, 300, 1, 33, 500], bw)
    ra, rb = random_tasks(rng, 150, bw)
    try:
        ctx.set_option("ungapped", 0)
        ctx.set_option("sw_form", form)
        for tb in (True, False):
            check_same(ctx.align(qs + ra, ts + rb, tb, D.ScoreParams(*scheme)), port.align(qs + ra, ts + rb, tb, scheme),
                       tb)
    finally:
        ctx.set_option("sw_form", 0)
        ctx.set_option("ungapped", 1)


@pytest.mark.parametrize("bw,n", [(8, 300), (8, 17_000), (16, 300), (16, 8_192), (16, 8_200), (64, 2_000), (64, 2_100),
                                  (21, 300)])
def test_windows_with_n_match_port(ctx, port, bw, n):
    """Tasks of the int32 kernel: an N in every target window, lists on both sides of the length
    from which it takes more cells a lane."""
    rng = np.random.default_rng(bw + n)
    sc = (2, 4, 4, 2, 1, bw)
    qs, ts = short_tasks(rng, rng.integers(1, 80, 300), bw)
    for q, t in zip(qs, ts):
        t[int(rng.integers(len(q)))] = 4
    times = -(-n // len(qs))
    want = (port.align(qs, ts, True, sc) * times)[:n]
    try:
        ctx.set_option("ungapped", 0)
        check_same(ctx.align((qs * times)[:n], (ts * times)[:n], True, D.ScoreParams(*sc)), want, True)
    finally:
        ctx.set_option("ungapped", 1)


@pytest.mark.parametrize("times", [1, 70])
def test_walks_over_long_runs_of_free_mismatches(ctx, port, times):
    """Mismatches that cost nothing fill every row a walk takes at once, in lists on both sides
    of the length up to which a task has a warp."""
    rng = np.random.default_rng(21)
    sc = (2, 0, 4, 2, 0, 16)
    qs, ts = [], []
    for i in range(90):
        core = rng.integers(0, 4, 700 + i).astype(np.uint8)
        q = core.copy()
        a, m = 40 + 3 * (i % 30), 100 + 6 * i
        q[a:a + m] = 4 if i % 2 else (q[a:a + m] + 1) % 4
        q = q[:len(q) - 16]
        s = int(rng.integers(0, 33))
        qs.append(q)
        ts.append(np.concatenate([rng.integers(0, 4, s).astype(np.uint8), core,
                                  rng.integers(0, 4, 40).astype(np.uint8)]))
    want = port.align(qs, ts, True, sc) * times
    try:
        ctx.set_option("ungapped", 0)
        check_same(ctx.align(qs * times, ts * times, True, D.ScoreParams(*sc)), want, True)
    finally:
        ctx.set_option("ungapped", 1)
