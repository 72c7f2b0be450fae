"""The int32 banded SW kernel on alignments that end about and beyond row 2^20, and whose scores
pass 2^24, against the oracle: the lanes of an alignment agree on the best row and column whatever
its row and score. Every task has gaps, so the DP runs."""
import numpy as np
import pytest

import dnaln_b200 as D
from test_gpu_align import check_same

pytestmark = pytest.mark.gpu


def gapped_task(rng, rows, bw):
    """A query of `rows` bases that aligns to its last base, with a gap every 50,000 or so."""
    t = rng.integers(0, 4, rows + 200).astype(np.uint8)
    cuts = np.sort(rng.integers(1000, rows - 1000, max(2, rows // 50_000)))
    q, at, shift = [], 0, 0
    for x in cuts:
        q.append(t[at:x])
        at = x + (1 if shift < bw // 2 else 0)  # a deletion, or an insertion once they add up
        if shift >= bw // 2:
            q.append(np.array([(int(t[x]) + 2) % 4], np.uint8))
        shift += 1 if shift < bw // 2 else -1
    q.append(t[at:])
    return np.concatenate(q)[:rows], np.concatenate([rng.integers(0, 4, bw // 4).astype(np.uint8), t])


@pytest.mark.parametrize("bw,rows,traceback,scores", [
    (8, 1_048_574, False, (2, 4, 4, 2, 1)), (8, 1_048_575, False, (2, 4, 4, 2, 1)),
    (8, 1_048_576, False, (2, 4, 4, 2, 1)), (8, 1_100_003, False, (2, 4, 4, 2, 1)),
    (8, 1_100_003, True, (2, 4, 4, 2, 1)), (8, 600_001, True, (40, 60, 60, 20, 1)),
    (16, 1_100_003, False, (2, 4, 4, 2, 1)), (16, 600_001, False, (40, 60, 60, 20, 1)),
    (32, 1_100_003, False, (2, 4, 4, 2, 1)), (64, 1_100_003, False, (2, 4, 4, 2, 1)),
])
def test_best_cell_beyond_row_2_to_20(ctx, port, bw, rows, traceback, scores):
    rng = np.random.default_rng(rows + bw)
    q, t = gapped_task(rng, rows, bw)
    want = port.align([q], [t], True, (*scores, bw))
    assert want[0][2] == rows and len(want[0][6]) > 1 and want[0][0] > rows
    check_same(ctx.align([q], [t], traceback, D.ScoreParams(*scores, bw)), want, traceback)
