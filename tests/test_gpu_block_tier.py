"""The block tier at the edges of its three shared-memory sizes (4096, 8192 and 16384 candidates a
side) and beyond the largest: one read whose end that many other reads continue, along one path that
each leaves at a place of its own, so that prefixes, equal continuations and strangers all occur.
The reference's method on the GPU (seed mode 0: walk + FM-index DFS, no block tier) gives the
expected graph; every field is a whole number, compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq

pytestmark = pytest.mark.gpu

L, T = 60, 20


def _fan(m, side, seed):
    rng = np.random.default_rng(seed)
    acgt = np.arange(1, 5, dtype=np.uint8)
    root, path = acgt[rng.integers(0, 4, L)], acgt[rng.integers(0, 4, L)]
    seen, rows = set(), [root]
    while len(rows) <= m:
        l = int(rng.integers(T, 46))
        r = np.concatenate([root[L - l:], path[:L - l]])
        p = int(rng.integers(l, L + 1))
        r[p:] = acgt[rng.integers(0, 4, L - p)]
        if r.tobytes() not in seen:
            seen.add(r.tobytes())
            rows.append(r)
    rd = np.stack(rows)
    if side:
        rd = 5 - rd[:, ::-1]
    return np.ascontiguousarray(rd[rng.permutation(len(rd))])


@pytest.mark.parametrize("width,side", [(32, 0), (64, 1)])
@pytest.mark.parametrize("m", [300, 4095, 4096, 4097, 8191, 8192, 8193, 16383, 16384, 16385])
def test_sides_at_the_edges_of_a_size(m, width, side):
    rd = _fan(m, side, m)
    out = {}
    for mode in (0, 1):
        with pq.Pasqual(width) as P:
            P.set_reads(rd, T)
            P.set_seed_mode(mode)
            P.build_index()
            out[mode] = P.construct_string_graph()
            tiers = P.tier_stats()
    assert tiers["deferred"] >= 1, tiers
    assert tiers["block"] >= 1 or m == 300, tiers
    for f in ("edge_off", "dest", "length", "etype", "trans", "num_B", "num_F", "olp_B", "olp_F"):
        assert np.array_equal(getattr(out[0], f), getattr(out[1], f)), f
