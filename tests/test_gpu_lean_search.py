"""The lean search tier against the oracle where its row selection changes branch: k-mers of few and
of many rows (seed depths down to 6 leave hundreds), rows narrowed by fewer bases than are kept
(t - k small), runs beyond the direct check, both continuation widths, reads that do not fill a warp.
Every output is a whole number: compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from oracle import port
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

SETS = {
    "L100": (dict(length=30_000, gc=0.42, repeat_frac=0.15, divergence=(0.005, 0.02), seed=51), 100, 20, 0.005, 63),
    "L100_t12": (dict(length=4_000, gc=0.5, seed=52), 100, 12, 0.002, 12),
    "L61_t31": (dict(length=20_000, gc=0.4, repeat_frac=0.1, seed=53), 61, 33, 0.01, 31),
    "L150_runs": (dict(length=20_000, gc=0.4, lowcomplex_frac=0.05, seed=54), 150, 18, 0.003, 63),
    "L233": (dict(length=20_000, gc=0.45, repeat_frac=0.3, divergence=(0.0, 0.01), seed=55), 233, 25, 0.01, 95),
    "L250_t31": (dict(length=8_000, gc=0.45, seed=56), 250, 14, 0.004, 31),
}


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("k", [0, 6, 8, 11])
@pytest.mark.parametrize("name", list(SETS))
def test_rows_selected_give_the_oracles_graph(name, k, width):
    shape, L, cov, err, t = SETS[name]
    gen = synth.genome(**shape)
    rd = synth.dedup(synth.reads_for_coverage(gen, L, cov, err, seed=61))
    rd = rd[: len(rd) - (len(rd) % 32 == 0)]
    O = port.Port(width)
    ref = O.overlaps(O.build_index(rd, t))
    with pq.Pasqual(width) as P:
        if k:
            P.set_seed_k(k)
        P.construct_index(rd, t)
        out = P.construct_string_graph()
    for f in ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans"):
        assert np.array_equal(getattr(out, f), getattr(ref, f)), f


@pytest.mark.parametrize("count", [3, 33, 4_000, 30_000, 60_000, 120_000, 200_000])
def test_reads_a_warp_by_their_number(count):
    """A warp takes 4 to 32 reads by the number of reads: the graph is the walk's (seed mode 0)."""
    gen = synth.genome(length=400 + count * 3, gc=0.45, repeat_frac=0.1, divergence=(0.0, 0.02), seed=71)
    rd = synth.dedup(synth.reads_for_coverage(gen, 60, 22, 0.003, seed=72))[:count]
    out = {}
    for mode in (0, 1):
        with pq.Pasqual(32) as P:
            P.set_reads(rd, 30)
            P.set_seed_mode(mode)
            P.build_index()
            out[mode] = P.construct_string_graph()
    for f in ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans"):
        assert np.array_equal(getattr(out[0], f), getattr(out[1], f)), f
