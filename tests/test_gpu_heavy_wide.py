"""The tiers behind the others where they take few reads: the heavy tier's groups of 4 to 32 reads a warp and the
wide tier's one read a warp, on reads whose continuations are too long for the sorted reduction, against the
oracle; whole numbers, compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from oracle import port
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("count", [33, 700, 4_000])
def test_few_reads_for_the_last_tiers(count, width):
    gen = synth.genome(length=60 + 12 * count, gc=0.41, repeat_frac=0.0, lowcomplex_frac=0.06, seed=3 + count)
    rd = synth.dedup(synth.reads_for_coverage(gen, 320, 27, 0.002, seed=4 + count)) if count > 33 else \
        synth.dedup(synth.reads_for_coverage(gen, 320, 40, 0.0, seed=4))
    O = port.Port(width)
    ref = O.overlaps(O.build_index(rd, 30))
    with pq.Pasqual(width) as P:
        P.construct_index(rd, 30)
        out = P.construct_string_graph()
        tiers = P.tier_stats()
    assert count == 33 or (tiers["heavy"] > 0 and tiers["wide"] > 0)
    for f in FIELDS:
        assert np.array_equal(getattr(out, f), getattr(ref, f)), f
