"""What a call that failed leaves behind: an index build that was refused after its k-mer table had been
cleared is no index, and a suffix array is kept where nothing of it was written."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("genome", [30_000, 300_000])
def test_a_refused_rebuild_is_no_index(genome, width):
    gen = synth.genome(length=genome, gc=0.42, repeat_frac=0.1, divergence=(0.0, 0.02), lowcomplex_frac=0.1, seed=41)
    rd = synth.dedup(synth.reads_for_coverage(gen, 100, 20, 0.003, seed=42))
    with pq.Pasqual(width) as P:
        P.construct_index(rd, 63)
        want, sa = P.construct_string_graph(), [P.get_sa(d) for d in (0, 1)]
        assert len(want.dest) > 0
        P.set_sort_chunk(max(2, rd.size // 2000))       # less than the one-base suffixes of a base
        with pytest.raises(pq.PQError) as refused:
            P.build_index()
        assert refused.value.code == 6
        with pytest.raises(pq.PQError) as unbuilt:
            P.overlaps()
        assert unbuilt.value.code == 5                  # PQ_ERR_STATE, not a graph without edges
        assert np.array_equal(P.get_sa(0), sa[0])       # the refusal comes before anything is sorted
        with pytest.raises(pq.PQError):
            P.sort(1)
        assert np.array_equal(P.get_sa(1), sa[1])
        P.set_sort_chunk(0)
        P.build_index()
        got = P.construct_string_graph()
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), getattr(want, f)), f


@pytest.mark.parametrize("L,reason", [(300, "268 bases"), (100, "6-base bucket")])
def test_a_refused_sort_names_its_reason(L, reason):
    gen = synth.genome(length=40_000, gc=0.42, seed=43)
    rd = synth.dedup(synth.reads_for_coverage(gen, L, 15, 0.003, seed=44))
    with pq.Pasqual(32) as P:
        P.set_reads(rd, 63)
        P.set_sort_chunk(rd.size // 2 if L > 268 else max(2, rd.size // 2000))
        with pytest.raises(pq.PQError, match=reason) as refused:
            P.sort(0)
        assert refused.value.code == 6
