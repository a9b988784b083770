"""The occurrence blocks and reads_index at the edges of a 64-row block and a 65536-row superblock,
from the sort's symbols and without them, against the oracle.  Whole numbers: equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("nr,L", [(1, 13), (3, 21), (4, 16), (5, 13), (8, 16), (97, 33), (1023, 64), (1024, 64), (1025, 64), (2049, 32), (2100, 63)])
def test_blocks_at_their_edges(nr, L, width):
    rng = np.random.default_rng(nr * L)
    rd = rng.integers(1, 5, (2 * nr, L)).astype(np.uint8)
    rd[: nr // 3, : L - 2] = 1                          # runs: blocks of many or no `$` rows
    rd = np.unique(rd, axis=0)
    rd = np.ascontiguousarray(rd[rng.permutation(len(rd))[:nr]])
    O = port.Port(width)
    ix = O.build_index(rd, 10)
    with pq.Pasqual(width) as P:
        P.set_reads(rd, 10)
        for kept in (True, False):
            for d in (0, 1):
                P.sort(d)
                if not kept:
                    P.sort(1 - d)                       # the scratch of the last sort is another direction's
                P.build_fm(d)
                bm, smp, ri = P.index_ref(d)
                assert np.array_equal(bm, ix["bitmap%d" % d])
                assert np.array_equal(smp, ix["sample%d" % d])
                assert np.array_equal(ri, ix["reads_index%d" % d])
