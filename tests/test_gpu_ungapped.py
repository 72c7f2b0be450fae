"""SW tasks proved to align without a gap (k_sw_ungapped) against the oracle, bit for bit:
query lengths at the edges of its 32-row words, bands at the edges of its three widths,
scoring schemes at the edges of the proof's preconditions, and the targets that defeat a
proof which is not one (tandem repeats, shifted copies, two-letter sequences, close and
clipped mismatches, indels, Ns)."""
import numpy as np
import pytest

import dnaln_b200 as D
from test_gpu_align import check_same

pytestmark = pytest.mark.gpu

# (match, mismatch, gap_open, gap_ext): the default, mismatch = match + gap_ext and
# match + mismatch = gap_open + gap_ext at once, one past the second, unit costs
SCHEMES = [(2, 4, 4, 2), (1, 2, 2, 1), (3, 3, 5, 0), (2, 4, 5, 2), (1, 1, 1, 1), (2, 3, 2, 2)]


def adversarial_tasks(rng, n, bw, lengths):
    qs, ts = [], []
    for i in range(n):
        L = int(lengths[i % len(lengths)])
        letters = int(rng.choice([2, 3, 4, 4, 4]))
        t = rng.integers(0, letters, L + 2 * bw).astype(np.uint8)
        kind = int(rng.integers(4))
        if kind == 1:  # a tandem repeat with a few errors
            period = int(rng.integers(1, 13))
            for j in range(period, len(t)):
                if rng.random() < 0.95:
                    t[j] = t[j - period]
        elif kind == 2:  # a stretch copied within the band
            a, m, s = int(rng.integers(len(t))), int(rng.integers(1, 60)), int(rng.integers(1, 2 * bw + 1))
            m = max(0, min(m, len(t) - a - s))
            t[a + s:a + s + m] = t[a:a + m].copy()
        q = t[bw:bw + L].copy()
        sub = rng.random(L) < rng.choice([0.0, 0.01, 0.03, 0.06])
        q[sub] = rng.integers(0, letters, int(sub.sum()))
        flaw = int(rng.integers(8))
        if flaw == 0:  # junk on an end or inside
            a = int(rng.integers(L))
            q[a:a + int(rng.integers(1, 20))] = rng.integers(0, letters)
        elif flaw == 1 and L > 4:  # a deletion, then an insertion elsewhere
            x, g = int(rng.integers(1, L)), int(rng.integers(1, 4))
            src = np.minimum(np.arange(x, L) + bw + g, len(t) - 1)
            q[x:] = t[src]
        elif flaw == 2 and L > 4:
            x, g = int(rng.integers(1, L)), int(rng.integers(1, 4))
            src = np.maximum(np.arange(x, L) + bw - g, 0)
            q[x:] = t[src]
        elif flaw == 3:  # an N in the query or the window, or a window cut short
            if rng.integers(2):
                q[int(rng.integers(L))] = 4
            else:
                t[int(rng.integers(len(t)))] = 4
        elif flaw == 4 and rng.integers(4) == 0:
            t = t[:int(rng.integers(len(t) + 1))]
        qs.append(q)
        ts.append(t)
    return qs, ts


@pytest.mark.parametrize("bw", [1, 5, 16, 17, 21, 32, 33, 64])
@pytest.mark.parametrize("scheme", SCHEMES)
def test_ungapped_tasks_match_port(ctx, port, scheme, bw):
    rng = np.random.default_rng(1000 * bw + 10 * scheme[1] + scheme[2])
    lengths = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 150, 160, 255, 256, 257]
    qs, ts = adversarial_tasks(rng, 1500, bw, lengths)
    sc = (*scheme, 1, bw)
    for tb in (True, False):
        check_same(ctx.align(qs, ts, tb, D.ScoreParams(*sc)), port.align(qs, ts, tb, sc), tb)


def test_ungapped_option_off_gives_the_same(ctx):
    rng = np.random.default_rng(5)
    qs, ts = adversarial_tasks(rng, 3000, 16, [50, 150, 151, 300, 999, 1000])
    sp = D.ScoreParams(2, 4, 4, 2, 1, 16)
    got = []
    try:
        for on in (1, 0):
            ctx.set_option("ungapped", on)
            got.append(ctx.align(qs, ts, True, sp))
    finally:
        ctx.set_option("ungapped", 1)
    for f in ("score", "qb", "qe", "tb", "te", "nm", "cigar_off", "cigar_len"):
        assert np.array_equal(got[0].results[f], got[1].results[f])
    assert np.array_equal(got[0].cigar, got[1].cigar)
