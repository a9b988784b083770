"""The suffix sort and the k-mer table it leaves, on inputs that reach each of its branches: one and
two partition passes, short suffixes sorted apart, buckets beyond either local kernel, groups equal
in all bases of their elements (33..128, ..1024, more, in one round and in several), chunks, networks
of every width and prefix doubling.  Suffix arrays and row numbers are whole numbers: compared for
equality with the oracle (oracle/pq_oracle.c)."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from oracle import port
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu


def iid(nr, L, seed, bases=4):
    return np.random.default_rng(seed).integers(1, bases + 1, (nr, L), dtype=np.uint8)


def covered(glen, L, cov, seed, err=0.003, runs=0.0, gc=0.42):
    return synth.reads_for_coverage(synth.genome(glen, gc, 0.1, (0.01, 0.02), runs, seed=seed), L, cov, err, seed=seed + 1)


def copies(kinds, times, L, seed):
    """`times` copies of each of `kinds` reads, with a few one-base changes."""
    rd = np.repeat(iid(kinds, L, seed), times, axis=0)
    rng = np.random.default_rng(seed + 1)
    for r in rng.integers(0, len(rd), len(rd) // 20):
        rd[r, rng.integers(0, L)] = rng.integers(1, 5)
    return rd[rng.permutation(len(rd))]


SHAPES = {
    # one pass (under 4 M suffixes), tiny to its largest
    "two_reads": (lambda: iid(2, 11, 1), 10, 0),
    "shortest_reads": (lambda: iid(3000, 11, 2), 10, 0),
    "one_pass": (lambda: covered(40_000, 100, 25, 3), 63, 0),
    "skewed": (lambda: covered(60_000, 75, 25, 4, gc=0.15), 31, 0),
    "two_bases": (lambda: iid(2500, 90, 5, bases=2), 40, 0),
    # two passes, with short suffixes sorted apart (44 K reads: one to three bases)
    "two_passes": (lambda: covered(180_000, 101, 25, 6), 47, 0),
    "short_suffixes": (lambda: iid(120_000, 40, 7), 31, 0),
    # groups of suffixes equal in all bases of their elements
    "groups_to_128": (lambda: copies(60, 90, 100, 8), 50, 0),
    "groups_to_1024": (lambda: copies(9, 700, 80, 9), 40, 0),
    "groups_beyond_1024": (lambda: copies(3, 3000, 120, 10), 60, 0),
    "all_equal": (lambda: np.full((9000, 60), 2, np.uint8), 30, 0),
    "poly_a_and_t": (lambda: np.where(iid(12_000, 50, 11) > 3, 4, 1).astype(np.uint8), 25, 0),
    "dinucleotide_runs": (lambda: covered(60_000, 150, 20, 12, runs=0.5), 63, 0),
    # network words by read length; prefix doubling beyond
    "L230": (lambda: covered(20_000, 230, 20, 13, err=0.01), 95, 0),
    "L262": (lambda: covered(20_000, 262, 15, 14, err=0.02), 95, 0),
    "L285": (lambda: covered(12_000, 285, 12, 15), 95, 0),
    "L301": (lambda: covered(12_000, 301, 12, 16), 95, 0),
    # sorted in chunks where one pass would need more memory than chunks of that size
    "chunks_of_a_sixth": (lambda: covered(60_000, 100, 25, 17), 63, 6),
    "chunks_two_passes": (lambda: covered(180_000, 101, 25, 18), 47, 40),
    "chunks_of_runs": (lambda: covered(60_000, 150, 20, 19, runs=0.3), 63, 12),
}


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("name", list(SHAPES))
def test_sort_and_kmers(name, width):
    make, t, parts = SHAPES[name]
    rd = np.ascontiguousarray(make())
    n = rd.size
    O = port.Port(width)
    with pq.Pasqual(width) as P:
        P.set_reads(rd, t)
        if parts:
            P.set_sort_chunk(n // parts)
        P.build_index()
        for d in (0, 1):
            want = O.sort(rd, d)
            assert np.array_equal(P.get_sa(d), want), d
            k = int(P.seeds(d)[2][0])
            ks, kz = O.kmer_table(rd, d, want, k)
            for got, ref in zip(P.seeds(d), O.seeds_from_kmers(rd, k, ks, kz, d)):
                assert np.array_equal(got, ref), d
            bm, smp, ri = P.index_ref(d)
            _, sfx, pfx = P.counts()
            for got, ref in zip((bm, smp, ri), O.build_occ(rd, d, want, pfx if d else sfx)):
                assert np.array_equal(got, ref), d
        P.sort(0)                                   # the suffix array alone
        assert np.array_equal(P.get_sa(0), O.sort(rd, 0))


@pytest.mark.parametrize("k", [1, 3, 7, 12])
def test_kmers_that_span_buckets(k):
    """k-mers shorter than the partition's own prefix, in one and in two passes."""
    for rd in (covered(40_000, 100, 25, 21), covered(180_000, 101, 25, 22), np.full((9000, 60), 2, np.uint8)):
        O = port.Port(32)
        with pq.Pasqual(32) as P:
            P.set_reads(rd, 40)
            P.set_seed_k(k)
            P.build_index()
            for d in (0, 1):
                ks, kz = O.kmer_table(rd, d, O.sort(rd, d), k)
                for got, ref in zip(P.seeds(d), O.seeds_from_kmers(rd, k, ks, kz, d)):
                    assert np.array_equal(got, ref), d
