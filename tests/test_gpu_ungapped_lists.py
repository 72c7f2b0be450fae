"""The proof of SW tasks without a gap in lists of every length (option "ungapped" 2) against the
oracle, and the lengths from which it runs by itself against the lists without it."""
import numpy as np
import pytest

import dnaln_b200 as D
from test_gpu_align import check_same
from test_gpu_ungapped import SCHEMES, adversarial_tasks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bw", [1, 5, 8, 16, 17, 21, 32, 33, 64])
@pytest.mark.parametrize("scheme", SCHEMES)
def test_proved_tasks_match_port(ctx, port, scheme, bw):
    rng = np.random.default_rng(1000 * bw + 10 * scheme[1] + scheme[2])
    lengths = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 150, 160, 255, 256, 257]
    qs, ts = adversarial_tasks(rng, 1500, bw, lengths)
    sc = (*scheme, 1, bw)
    try:
        ctx.set_option("ungapped", 2)
        for tb in (True, False):
            check_same(ctx.align(qs, ts, tb, D.ScoreParams(*sc)), port.align(qs, ts, tb, sc), tb)
    finally:
        ctx.set_option("ungapped", 1)


@pytest.mark.parametrize("bw,limit", [(5, 10_240), (8, 14_336), (16, 7_168), (21, 2_560), (32, 2_304), (64, 1_536)])
def test_lists_around_the_length_that_pays(ctx, port, bw, limit):
    rng = np.random.default_rng(bw)
    qs, ts = adversarial_tasks(rng, 300, bw, [20, 33, 64, 90])
    sc = (2, 4, 4, 2, 1, bw)
    want = port.align(qs, ts, True, sc)
    for n in (1, 4, 5, limit, limit + 1):
        times = -(-n // len(qs))
        ctx.set_kernel_trace(True)
        try:
            ctx.reset_stats()
            got = ctx.align((qs * times)[:n], (ts * times)[:n], True, D.ScoreParams(*sc))
            ran = "k_sw_ungapped<tb>" in ctx.kernel_times()
        finally:
            ctx.set_kernel_trace(False)
        check_same(got, (want * times)[:n], True)
        assert ran == (n <= 4 or n > limit)
