"""Contexts on different host threads at the same time, as the header allows: index builds and searches
of read sets whose sorts take partition passes of different widths and whose reads differ in length,
with reads for the block tier.  Every graph is the one the same set gives alone."""
import threading

import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")
SETS = [(300_000, 100, 20, 0.02, 63), (2_000, 60, 15, 0.05, 25), (60_000, 200, 18, 0.02, 95), (500, 45, 12, 0.1, 20)]


def test_builds_and_searches_of_four_threads():
    sets = []
    for i, (length, L, cov, runs, t) in enumerate(SETS):
        gen = synth.genome(length=length, gc=0.42, repeat_frac=0.1, divergence=(0.0, 0.02), lowcomplex_frac=runs, seed=91 + i)
        sets.append((synth.dedup(synth.reads_for_coverage(gen, L, cov, 0.003, seed=95 + i)), t))

    def search(rd, t):
        with pq.Pasqual(32) as P:
            P.construct_index(rd, t)
            return P.construct_string_graph()

    alone = [search(*s) for s in sets]
    faults = []

    def work(i):
        try:
            for _ in range(12):
                out = search(*sets[i])
                for f in FIELDS:
                    assert np.array_equal(getattr(out, f), getattr(alone[i], f)), (i, f)
        except Exception as e:                      # noqa: BLE001 (reported by the main thread)
            faults.append(repr(e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults, faults
