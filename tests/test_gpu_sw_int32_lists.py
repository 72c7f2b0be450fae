"""The int32 SW kernel's two forms on both sides of the list length that divides them, against the
oracle: every window has an N."""
import numpy as np
import pytest

import dnaln_b200 as D
from test_gpu_align import check_same
from test_gpu_sw_forms import short_tasks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bw,limit", [(8, 12_288), (16, 6_144), (32, 3_072), (64, 1_536)])
def test_lists_around_the_forms_limit(ctx, port, bw, limit):
    rng = np.random.default_rng(bw)
    sc = (2, 4, 4, 2, 1, bw)
    qs, ts = short_tasks(rng, rng.integers(1, 80, 250), bw)
    for q, t in zip(qs, ts):
        t[int(rng.integers(len(q)))] = 4
    want = port.align(qs, ts, True, sc)
    for n in (limit, limit + 1):
        times = -(-n // len(qs))
        for tb in (True, False):
            check_same(ctx.align((qs * times)[:n], (ts * times)[:n], tb, D.ScoreParams(*sc)), (want * times)[:n], tb)
