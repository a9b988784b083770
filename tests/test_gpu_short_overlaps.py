"""Overlaps so short that an ordinary read's depth-t interval outgrows the interval scan by chance: enough
such reads go to the fast tier, the rest to the block tier, alone and as a set of a batch.  The graph is
that of seed mode 0, which walks every read; whole numbers, compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")


def context(rd, width, mode):
    P = pq.Pasqual(width)
    P.set_seed_mode(mode)
    P.construct_index(rd, 10)
    return P


# rows / 4^10 of 31 to 63 at a GC content that skews the k-mers: few misses and many, some of them of more than
# 64 candidates a side; both widths of the continuation
@pytest.mark.parametrize("width,genome,gc,runs,L", [(32, 1_500_000, 0.36, 0.0, 100), (32, 3_000_000, 0.36, 0.0, 250), (64, 2_800_000, 0.38, 0.0002, 180),
                                                    (32, 1_850_000, 0.42, 0.0, 74)])
def test_misses_by_chance(width, genome, gc, runs, L):
    gen = synth.genome(length=genome, gc=gc, lowcomplex_frac=runs, seed=91)
    rd = synth.dedup(synth.reads_for_coverage(gen, L, 22, 0.003, seed=92))
    with context(rd, width, 0) as P:
        want = P.construct_string_graph()
    small = rd[:5_000]
    with context(rd, width, 1) as P, context(small, width, 1) as Q, context(small, width, 0) as R:
        got = P.construct_string_graph()
        tiers = P.tier_stats()
        again = P.construct_string_graph()          # the edge pool has grown
        pq.overlaps_batched([Q, P])
        batched, other, ref = P.graph(), Q.graph(), R.construct_string_graph()
    assert tiers["deferred"] > 0
    assert tiers["deferred"] < 16384 or tiers["block"] < tiers["deferred"]
    for f in FIELDS:
        for x in (got, again, batched):
            assert np.array_equal(getattr(x, f), getattr(want, f)), f
        assert np.array_equal(getattr(other, f), getattr(ref, f)), f
