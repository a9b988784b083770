"""The sort's seed records on buckets that span several levels of the minima they are found by (64,
4096 and 262144 rows): reads of long single-base runs.  Expected: the reference's rule, depth by depth
over the suffix array (a bucket of more than one suffix records for the suffixes of exactly its depth;
it is recursed into at depth 9, or with size * (L - D + 3) >= 3500).  Whole numbers: equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq

pytestmark = pytest.mark.gpu


def _expected(reads, sa, t, seeds):
    nr, L = reads.shape
    n, dmax = nr * L, 3 * (t // 3)
    start, size, depth = (a.copy() for a in seeds)
    text = np.concatenate([reads.reshape(-1), np.zeros(dmax, np.uint8)])
    r, off = sa // L, sa % L
    length = L - off
    rows = np.zeros((n, dmax), np.uint8)
    for j in range(dmax):
        rows[:, j] = np.where(length > j, text[sa + j], 0)
    same = (rows[1:] == rows[:-1]) & (rows[1:] != 0)
    lcp = np.concatenate([[0], np.where(same.all(1), dmax, (~same).argmax(1))])
    parent = np.ones(n, bool)
    for D in range(9, dmax + 1, 3):
        head = lcp < D
        first = np.flatnonzero(head)
        which = np.cumsum(head) - 1
        sizes = np.diff(np.append(first, n))
        visited = parent[first] & (sizes > 1)
        rec = visited[which] & (length == D) & (depth[r] < D)
        depth[r[rec]], start[r[rec]], size[r[rec]] = D, first[which[rec]], sizes[which[rec]]
        parent = (visited & ((D == 9) | (sizes * (L - D + 3) >= 3500)))[which]
    return start, size, depth


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("nr,L,t", [(5, 30, 10), (40, 30, 21), (700, 33, 23), (9000, 60, 21), (3000, 101, 63)])
def test_buckets_of_long_runs(nr, L, t, width):
    rng = np.random.default_rng(nr + L)
    rd = np.ones((nr, L), np.uint8)
    for _ in range(3):
        rd[np.arange(nr), rng.integers(0, L, nr)] = rng.integers(1, 5, nr)
    rd[:, : L // 4] = np.where(rng.random((nr, 1)) < 0.5, rng.integers(1, 5, (nr, L // 4)), rd[:, : L // 4])
    rd = np.ascontiguousarray(np.unique(rd, axis=0).astype(np.uint8))
    with pq.Pasqual(width) as P:
        P.set_reads(rd, t)
        P.sort(0)
        sa = P.get_sa(0).astype(np.int64)
        got = P.sort_seeds(0)
    n = len(rd)
    last = rd[:, -1]
    counts = np.concatenate([[0], np.cumsum(np.bincount(rd.reshape(-1), minlength=5)[1:])])
    init = (counts[last - 1].astype(np.int64), np.bincount(rd.reshape(-1), minlength=5)[last].astype(np.int64), np.ones(n, np.int64))
    want = _expected(rd, sa, t, init)
    for g, w, what in zip(got, want, ("start", "size", "depth")):
        assert np.array_equal(np.asarray(g).astype(np.int64), w), what
