"""The sort in chunks: runs of first-level buckets of one pass over the text, and a pass over the text for
every chunk where a first-level bucket is larger than a chunk.  Suffix arrays, k-mer rows and FM-indexes
are those of the sort in one piece (compared with the oracle elsewhere), for few and many chunks, ordinary
and low-complexity reads, k-mers within and across buckets; whole numbers, compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu


def _reads(name):
    if name == "equal":
        return np.full((45_000, 100), 3, np.uint8)
    shape = {"plain": dict(gc=0.42, repeat_frac=0.1, divergence=(0.0, 0.02)), "runs": dict(gc=0.42, lowcomplex_frac=0.3),
             "skewed": dict(gc=0.1)}[name]
    return synth.reads_for_coverage(synth.genome(length=400_000, seed=31, **shape), 101, 25, 0.003, seed=32)


def _index(P, k):
    out = []
    for d in (0, 1):
        out += [P.get_sa(d), *P.seeds(d), *P.index_ref(d)]
    return out


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("name,k", [("plain", 0), ("plain", 3), ("runs", 0), ("skewed", 7), ("equal", 0)])
def test_chunks_give_the_sort_in_one_piece(name, k, width):
    rd = _reads(name)
    n = rd.size
    refused = 0
    with pq.Pasqual(width) as P:
        if k:
            P.set_seed_k(k)
        P.construct_index(rd, 47)
        want = _index(P, k)
        for parts in (6, 13, 50, 250):
            P.set_sort_chunk(n // parts)
            try:
                P.build_index()
            except pq.PQError as e:         # a bucket of six bases larger than a chunk
                assert e.code == 6
                refused += 1
                continue
            for got, ref in zip(_index(P, k), want):
                assert np.array_equal(got, ref), parts
    assert refused == 0 or name != "plain"
