"""Seed depths at which suffixes of a few bases, sorted apart, lie inside k-mers (depth 4 from about
131 K reads on): their rows' next bases are those of this read set, not what an earlier index of the
same context left there.  The graph is the walk's (seed mode 0), which uses no such rows; whole numbers,
compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")


def _reads(seed, count, gc, L=50):
    gen = synth.genome(length=count * 3, gc=gc, repeat_frac=0.1, divergence=(0.0, 0.02), seed=seed)
    return synth.dedup(synth.reads_for_coverage(gen, L, 20, 0.003, seed=seed + 1))[:count]


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("k", [3, 4])
def test_graph_at_a_depth_below_the_short_suffixes(k, width):
    before, rd = _reads(81, 150_000, 0.6), _reads(83, 149_000, 0.42)
    assert len(rd) >> (2 * k) > 512 and len(rd[0]) >= 4 * k
    out = {}
    with pq.Pasqual(width) as P:
        P.set_seed_k(k)
        for mode in (0, 1):
            P.set_seed_mode(mode)
            P.construct_index(before, 31)               # another set's rows where this one's will be
            P.construct_index(rd, 31)
            out[mode] = P.construct_string_graph()
    for f in FIELDS:
        assert np.array_equal(getattr(out[0], f), getattr(out[1], f)), f
