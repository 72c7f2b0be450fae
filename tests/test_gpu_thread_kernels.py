"""The thread-per-read seeding kernels against the oracle where they really run: more reads than a
list that is handed on unread, with every read theirs (option "colinear" 0), and with a list of
the reads the colinear check left."""
import numpy as np
import pytest

import dnaln_b200 as D
from dnaln_b200 import synth
from test_gpu_colinear import genome, make_reads
from test_gpu_map import assert_same_as

pytestmark = pytest.mark.gpu

HANDED_ON = 4096  # lists of at most this many reads go to the warp kernels as they are


def check(ctx, port, g, reads, colinear, **options):
    iid = ctx.index_build(g)
    rec = port.map(port.index(g), reads, D.default_map_params())
    stats = []
    try:
        ctx.set_option("colinear", colinear)
        for values in zip(*options.values()) if options else [()]:
            for o, v in zip(options, values):
                ctx.set_option(o, v)
            ctx.reset_stats()
            assert_same_as(rec, ctx.map_batch(iid, reads), len(reads))
            stats.append(ctx.stats())
    finally:
        ctx.set_option("colinear", 1)
        ctx.set_option("seed_block", 0)
        ctx.set_option("long_thread", 1)
        ctx.index_free(iid)
    return stats


def many(reads, times):
    seqs = [reads.read(i) for i in range(len(reads))] * times
    return D.ReadBatch.from_lists(seqs, [b"r%d" % i for i in range(len(seqs))])


def test_every_block_size_on_all_reads(ctx, port):
    rng = np.random.default_rng(1)
    g = genome(rng)
    reads = many(make_reads(rng, g, 2_000, [30, 64, 100, 149, 150, 151]), 4)
    for st in check(ctx, port, g, reads, 0, seed_block=(64, 128)):
        assert st["warp_reads"] < len(reads) // 4  # the thread kernel finished most


def test_long_reads_on_all_reads(ctx, port):
    rng = np.random.default_rng(2)
    g = genome(rng)
    reads = many(make_reads(rng, g, 1_500, [300, 420, 500, 800, 1000]), 4)
    on, off = check(ctx, port, g, reads, 0, long_thread=(1, 0))
    # without the colinear kernels the counter is the long-read thread kernel's alone
    assert on["long_reads"] > len(reads) // 2 and off["long_reads"] == 0
    assert off["warp_reads"] - on["warp_reads"] == on["long_reads"]


@pytest.mark.parametrize("lengths", [[60, 100, 150, 151], [300, 500, 800]])
def test_listed_reads(ctx, port, lengths):
    """Chimeras and reads with a far copy: more of them than are handed on unread."""
    rng = np.random.default_rng(3)
    g = genome(rng)
    base = make_reads(rng, g, 3_000, lengths)
    seqs = [base.read(i) for i in range(len(base))]
    mixed = [a[:len(a) // 2] + b[len(b) // 2:] for a, b in zip(seqs, seqs[1:] + seqs[:1])]
    reads = D.ReadBatch.from_lists(mixed * 4, [b"r%d" % i for i in range(4 * len(mixed))])
    long = lengths[0] >= 300
    stats = check(ctx, port, g, reads, 1, **({"long_thread": (1, 0)} if long else {"seed_block": (64, 128)}))
    listed = check(ctx, port, g, reads, 1, long_thread=(0,))[0]["warp_reads"] if long else None
    if long:
        assert listed > HANDED_ON and stats[0]["warp_reads"] < listed  # the thread kernel took some of the list


@pytest.mark.parametrize("n", [1, HANDED_ON, HANDED_ON + 1])
def test_long_lists_around_the_length_that_is_handed_on(ctx, port, n):
    rng = np.random.default_rng(4)
    g = genome(rng)
    reads = many(make_reads(rng, g, 1_100, [300, 420]), 4).slice(0, n)
    (st,) = check(ctx, port, g, reads, 0)
    assert (st["long_reads"] > 0) == (n > HANDED_ON)


@pytest.mark.parametrize("times,lengths", [(1, [100, 150]), (1, [150, 300, 600]), (5, [100, 150]), (5, [150, 300, 600])])
def test_reads_with_an_n(ctx, port, times, lengths):
    """Every read has an N, so none is sketched for the colinear check: lists that are handed on and
    lists the thread kernels take, with reads too rich in anchors for those."""
    rng = np.random.default_rng(5)
    g = genome(rng)
    base = make_reads(rng, g, 1_000, lengths)
    seqs = []
    for i in range(len(base)):
        q = bytearray(base.read(i))
        if i % 4 == 0:  # inside the tandem repeat
            at = 60_000 + i % 30
            q = bytearray(b"ACGTN"[c] for c in g.codes[at:at + min(len(q), 440)])
        q[int(rng.integers(len(q)))] = ord("N")
        seqs.append(bytes(q))
    reads = D.ReadBatch.from_lists(seqs * times, [b"r%d" % i for i in range(times * len(seqs))])
    on, off = check(ctx, port, g, reads, 1)[0], check(ctx, port, g, reads, 0)[0]
    for f in ("mapped", "candidates", "minimizers", "anchors"):
        assert on[f] == off[f], f
    assert 0 < on["warp_reads"] and (on["warp_reads"] == len(reads)) == (times == 1)
