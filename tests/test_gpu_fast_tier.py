"""The fast tier (seed mode 0: FM-index walk and DFS) against the oracle where its reduction changes
branch: levels of up to 32 intervals (sets counted by ballots) and of more (bit masks), tasks that
do not fill a warp's queue, reads without candidates between others.  Every output is a whole number:
compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from oracle import port
from pasqual_gb300 import synth

pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")


def _check(rd, t, width):
    O = port.Port(width)
    ref = O.overlaps(O.build_index(rd, t))
    with pq.Pasqual(width) as P:
        P.set_reads(rd, t)
        P.set_seed_mode(0)
        P.build_index()
        out = P.construct_string_graph()
    for f in FIELDS:
        assert np.array_equal(getattr(out, f), getattr(ref, f)), f


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("groups", [1, 16, 31, 32, 33, 48, 63, 64])
def test_levels_of_so_many_intervals(groups, width):
    """One read whose end `groups` reads continue, each from an overlap length of its own (an interval
    each), along one path that some of them leave; the same reads complemented double the intervals."""
    L, t = 100, 20
    rng = np.random.default_rng(groups)
    root, path = rng.integers(1, 5, L).astype(np.uint8), rng.integers(1, 5, L).astype(np.uint8)
    rows = [root]
    for l in range(t, t + groups):
        r = np.concatenate([root[L - l:], path[:L - l]])
        p = int(rng.integers(l, 2 * L))
        r[p:] = rng.integers(1, 5, max(L - p, 0))
        rows.append(r)
    rd = np.stack(rows)
    _check(rd, t, width)
    both = np.concatenate([rd, 5 - rd[1:, ::-1]])
    _check(np.ascontiguousarray(np.unique(both, axis=0)), t, width)


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 95, 127, 128, 129, 161, 700])
def test_queues_of_so_many_reads(count, width):
    gen = synth.genome(length=1 + count * 6, gc=0.45, repeat_frac=0.2, seed=count) if count > 40 else synth.genome(length=300, gc=0.45, seed=count)
    rd = synth.dedup(synth.reads_for_coverage(gen, 60, 40, 0.005, seed=7))[:count]
    rd = np.concatenate([rd, np.random.default_rng(count).integers(1, 5, (max(count - len(rd), 0), 60)).astype(np.uint8)])
    _check(np.ascontiguousarray(rd[np.random.default_rng(1).permutation(len(rd))]), 20, width)
