"""Partition buckets beyond the local kernels in their hundreds (skewed base composition, a few reads in
thousands of copies with errors): split on the device, their parts listed there.  The suffix array is checked
row by row in numpy (every suffix's bases as two 64-bit words, its length and its position in order), the k-mer
table entered by the sort against the one built from the suffix array."""
import numpy as np
import pytest

import pasqual_gb300 as pq

pytestmark = pytest.mark.gpu


def skewed(nr, L, gc, rng):
    return (rng.choice(4, size=(nr, L), p=[(1 - gc) / 2, gc / 2, gc / 2, (1 - gc) / 2]) + 1).astype(np.uint8)


def copies(kinds, times, L, err, rng):
    base = rng.integers(1, 5, (kinds, L), dtype=np.uint8)
    rd = base[rng.permutation(np.repeat(np.arange(kinds), times))]
    flip = rng.random(rd.shape, dtype=np.float32) < err
    return np.where(flip, rng.integers(1, 5, rd.shape, dtype=np.uint8), rd)


def suffix_words(rd, backward):
    """(two words of bases, length) of the suffix at every position, L <= 64."""
    t = (rd[:, ::-1] if backward else rd).astype(np.uint64) - 1
    nr, L = t.shape
    w = np.zeros((2, nr, L + 1), np.uint64)
    for o in range(L - 1, -1, -1):
        w[1, :, o] = (w[1, :, o + 1] >> np.uint64(2)) | ((w[0, :, o + 1] & np.uint64(3)) << np.uint64(62))
        w[0, :, o] = (w[0, :, o + 1] >> np.uint64(2)) | (t[:, o] << np.uint64(62))
    length = np.broadcast_to(np.arange(L, 0, -1, dtype=np.int64), (nr, L))
    return w[0, :, :L].ravel(), w[1, :, :L].ravel(), length.ravel()


# 32 kinds of 50 bases: 1,600 buckets of 12 thousand suffixes, 293 of which are split at a time, each with a part that
# is too large once more
@pytest.mark.parametrize("name", ["gc05", "gc25", "copies", "copies_few"])
@pytest.mark.parametrize("width", [32, 64])
def test_large_buckets(name, width):
    rng = np.random.default_rng(17)
    rd = {"gc05": lambda: skewed(250_000, 40, 0.05, rng), "gc25": lambda: skewed(600_000, 40, 0.25, rng),
          "copies": lambda: copies(32, 12_000, 50, 0.004, rng), "copies_few": lambda: copies(3, 30_000, 33, 0.002, rng)}[name]()
    with pq.Pasqual(width) as P:
        P.set_reads(rd, 20)
        P.set_seed_k(11)
        P.build_index()
        seeds = [P.seeds(d) for d in (0, 1)]
        for d in (0, 1):
            sa = P.get_sa(d).astype(np.int64)
            assert np.array_equal(np.bincount(sa, minlength=rd.size), np.ones(rd.size, np.int64))
            less = np.zeros(rd.size - 1, bool)
            tie = np.ones(rd.size - 1, bool)
            for x in (*suffix_words(rd, d == 1), np.arange(rd.size)):
                x = x[sa]
                less |= tie & (x[:-1] < x[1:])
                tie &= x[:-1] == x[1:]
            assert less.all()
            P.set_sa(d, P.get_sa(d))
            P.build_fm(d)
            assert all(np.array_equal(a, b) for a, b in zip(seeds[d], P.seeds(d)))
