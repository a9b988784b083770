"""The static sort on device buffers that start at any byte: both directions against the oracle's order
(whole numbers, compared for equality)."""
import numpy as np
import pytest

from oracle import port
from test_zz_no_alloc import static_sort_fn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("nr,L", [(1, 33), (3, 37), (40, 101), (7000, 100), (4001, 63)])
@pytest.mark.parametrize("shift", [1, 4, 7])
def test_reads_at_an_unaligned_address(nr, L, shift, width):
    import torch
    rd = np.random.default_rng(nr + L + shift).integers(1, 5, (nr, L), dtype=np.uint8)
    buf = torch.zeros(nr * L + shift, dtype=torch.uint8, device="cuda")
    buf[shift:] = torch.from_numpy(rd.reshape(-1)).cuda()
    sa = torch.empty(nr * L, dtype=torch.int64 if width == 64 else torch.int32, device="cuda")
    f, O = static_sort_fn(width), port.Port(width)
    for d in (0, 1):
        assert f(buf.data_ptr() + shift, nr, L, d, sa.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        assert np.array_equal(sa.cpu().numpy().view(O.sort(rd, d).dtype), O.sort(rd, d)), d
