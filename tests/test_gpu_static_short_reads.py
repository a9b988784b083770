"""The static sort (pq_suffix_sort_static takes any read length) on reads of 1 to 9 bases, where words
of the packed text span many reads, against numpy's stable sort by (bases, end of read lowest)."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from test_zz_no_alloc import static_sort_fn

pytestmark = pytest.mark.gpu


def _expected(reads, direction):
    nr, L = reads.shape
    text = (reads if direction == 0 else reads[:, ::-1]).reshape(-1)
    pos = np.arange(nr * L)
    left = L - pos % L
    cols = [np.where(left > j, text[np.minimum(pos + j, nr * L - 1)], 0) for j in range(L)]
    return np.lexsort([pos] + cols[::-1])


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("nr,L", [(1, 1), (33, 1), (20_000, 1), (200_000, 1), (5, 2), (70_000, 2), (60_000, 3), (30_000, 5), (4, 7), (20_000, 7), (9, 8), (30_001, 8), (20_000, 9)])
def test_reads_of_few_bases(nr, L, width):
    import torch
    rd = np.random.default_rng(nr + L).integers(1, 5, (nr, L), dtype=np.uint8)
    dev = torch.device("cuda", 0)
    reads = torch.from_numpy(rd).to(dev)
    sa = torch.empty(nr * L, dtype=torch.int64 if width == 64 else torch.int32, device=dev)
    f = static_sort_fn(width)
    for direction in (0, 1):
        assert f(reads.data_ptr(), nr, L, direction, sa.data_ptr(), torch.cuda.current_stream(dev).cuda_stream) == 0
        assert np.array_equal(sa.cpu().numpy(), _expected(rd, direction)), direction
