"""Groups of equal suffixes at the edges of the sort's kernels for them (128 and 1024 members, one CTA's
network over any number of places) and ranges split further by the host, whose parts are put together
up to a local kernel's 8192: sets of `times` copies of each of a few reads.  The oracle's suffix array;
whole numbers, compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("kinds,times", [(7, 129), (5, 200), (3, 511), (3, 513), (2, 1000), (2, 1024), (2, 1025), (1, 8192),
                                         (1, 8193), (2, 8191), (1, 20_000)])
def test_copies_of_a_few_reads(kinds, times, width):
    rng = np.random.default_rng(kinds * times)
    rd = np.repeat(rng.integers(1, 5, (kinds, 70), dtype=np.uint8), times, axis=0)
    rd = np.ascontiguousarray(rd[rng.permutation(len(rd))])
    O = port.Port(width)
    with pq.Pasqual(width) as P:
        P.set_reads(rd, 40)
        P.build_index()
        for d in (0, 1):
            assert np.array_equal(P.get_sa(d), O.sort(rd, d)), d
