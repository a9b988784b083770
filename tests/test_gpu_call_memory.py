"""Calls that take device memory for themselves give all of it back."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CALLS = {
    "sort_seeds": lambda P: P.sort_seeds(1),
    "seeds": lambda P: P.seeds(0),
    "index_ref": lambda P: P.index_ref(1),
    "learned_predict": lambda P: P.learned_predict(0, np.arange(1 << 22, dtype=np.uint32)),
}


@pytest.mark.parametrize("name", list(CALLS))
def test_memory_comes_back(name):
    gen = synth.genome(length=400_000, gc=0.42, seed=95)
    rd = synth.dedup(synth.reads_for_coverage(gen, 100, 20, 0.003, seed=96))
    with pq.Pasqual(32) as P:
        P.construct_index(rd, 63)
        P.learned_build(0, 5)
        CALLS[name](P)
        before = torch.cuda.mem_get_info()[0]
        for _ in range(4):                      # a leak of one call is megabytes, allocations being 2 MB each
            CALLS[name](P)
        assert torch.cuda.mem_get_info()[0] == before
