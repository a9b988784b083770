"""Reads of 10 to 16 bases, of which up to half the suffixes are short ones sorted apart: the suffix arrays
against numpy's sort by (bases, end of read lowest, position), by a context and, at the most it accepts, by the
static sort; the k-mer table entered by the sort against the one built from the suffix array."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from test_zz_no_alloc import static_sort_fn

pytestmark = pytest.mark.gpu


def expected(rd, direction):
    """Bases and length in one word: 2 bits a base, then 5 bits of length (reads of up to 29 bases)."""
    t = (rd if direction == 0 else rd[:, ::-1]).astype(np.int64) - 1
    nr, L = t.shape
    key = np.zeros((nr, L + 1), np.int64)
    for o in range(L - 1, -1, -1):
        key[:, o] = (key[:, o + 1] >> 2) | (t[:, o] << (2 * L - 2))
    return np.argsort(((key[:, :L] << 5) | np.arange(L, 0, -1)).ravel(), kind="stable")


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("L", [11, 12, 13, 15, 16])
@pytest.mark.parametrize("nr", [3_000, 560_000])        # 560 thousand: suffixes of up to 5 bases apart
def test_context(nr, L, width):
    rd = np.random.default_rng(L).choice(4, (nr, L), p=[0.3, 0.2, 0.2, 0.3]).astype(np.uint8) + 1
    with pq.Pasqual(width) as P:
        P.set_reads(rd, 10)
        for k in (4, 10):
            P.set_seed_k(k)
            P.build_index()
            for d in (0, 1):
                assert np.array_equal(P.get_sa(d).astype(np.int64), expected(rd, d)), d
                seeds = P.seeds(d)
                P.set_sa(d, P.get_sa(d))
                P.build_fm(d)
                assert all(np.array_equal(a, b) for a, b in zip(seeds, P.seeds(d))), d


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("L", [4, 6, 8, 9, 10, 11, 12, 14])
def test_static(L, width):
    import torch
    rd = np.random.default_rng(L).integers(1, 5, ((1 << 20) // L, L), dtype=np.uint8)
    reads = torch.from_numpy(rd).cuda()
    sa = torch.empty(rd.size, dtype=torch.int64 if width == 64 else torch.int32, device="cuda")
    f = static_sort_fn(width)
    for d in (0, 1):
        assert f(reads.data_ptr(), len(rd), L, d, sa.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        assert np.array_equal(sa.cpu().numpy(), expected(rd, d)), d
