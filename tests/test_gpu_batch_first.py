"""A batch is the first search of all its contexts, none of which has the scratch of a search of its own
yet: every graph is the one that another context gives alone."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")
SHAPES = [(40_000, 100, 20, 63, 0.0), (9_000, 61, 25, 31, 0.05), (30_000, 150, 18, 70, 0.02), (3_000, 45, 12, 20, 0.0),
          (60_000, 233, 20, 95, 0.0)]


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("count,use_graph", [(1, False), (2, True), (3, False), (5, True)])
def test_batch_of_contexts_never_searched(count, use_graph, mode):
    def contexts():
        out = []
        for i, (length, L, cov, t, runs) in enumerate(SHAPES[:count]):
            gen = synth.genome(length=length, gc=0.42, repeat_frac=0.1, divergence=(0.0, 0.02), lowcomplex_frac=runs, seed=61 + i)
            P = pq.Pasqual(32)
            P.set_seed_mode(mode)
            P.construct_index(synth.dedup(synth.reads_for_coverage(gen, L, cov, 0.003, seed=66 + i)), t)
            out.append(P)
        return out

    batch, alone = contexts(), contexts()
    try:
        pq.overlaps_batched(batch, graph=use_graph)
        for P, Q in zip(batch, alone):
            got, want = P.graph(), Q.construct_string_graph()
            for f in FIELDS:
                assert np.array_equal(getattr(got, f), getattr(want, f)), f
    finally:
        for P in batch + alone:
            P.close()
