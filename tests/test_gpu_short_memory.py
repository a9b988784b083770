"""Device memory that runs short: what a build or a search can do without (the rows' next bases, the sort's
working memory, a sort of everything at once) gives way to what it needs.  The card is filled with an
allocation of its own up to the room that is left; every output is a whole number, compared for equality."""
import numpy as np
import pytest

import pasqual_gb300 as pq
from pasqual_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FIELDS = ("num_B", "num_F", "olp_B", "olp_F", "edge_off", "dest", "length", "etype", "trans")
T, SEED_K = 63, 10


def free():
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def fill(left):
    """An allocation that leaves `left` bytes."""
    return torch.empty(free() - left, dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def reads():
    gen = synth.genome(length=2_000_000, gc=0.42, repeat_frac=0.1, divergence=(0.0, 0.02), seed=81)
    return synth.dedup(synth.reads_for_coverage(gen, 100, 20, 0.003, seed=82))


def context(rd, width):
    P = pq.Pasqual(width)
    P.set_reads(rd, T)
    P.set_seed_k(SEED_K)
    return P


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("less", [3, 8])        # bytes a suffix less than a build takes: kx is 4 of them
def test_a_build_with_less_memory(less, width, reads):
    with context(reads, width) as P:
        before = free()
        P.build_index()
        used = before - free()
        want, sa = P.construct_string_graph(), [P.get_sa(d) for d in (0, 1)]
    with context(reads, width) as P:
        hog = fill(used - less * reads.size)
        P.build_index()
        assert all(np.array_equal(P.get_sa(d), sa[d]) for d in (0, 1))
        del hog
        torch.cuda.empty_cache()
        got = P.construct_string_graph()
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), getattr(want, f)), f


@pytest.mark.parametrize("batch", [1, 3])
def test_a_search_with_less_memory(batch, reads):
    def search(ctxs):
        if batch > 1:
            pq.overlaps_batched(ctxs)
        else:
            ctxs[0].overlaps()

    parts = [reads] if batch == 1 else [reads[: 100_000 + 7], reads[: 50_001], reads]
    out = []
    for short in (False, True):
        ctxs = [context(rd, 32) for rd in parts]
        try:
            for P in ctxs:
                P.build_index()
            before = free()
            hog = fill(used - 3 * reads.size) if short else None
            search(ctxs)
            used = before - free()
            del hog
            out.append([P.graph() for P in ctxs])
        finally:
            for P in ctxs:
                P.close()
    for a, b in zip(*out):
        for f in FIELDS:
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


def test_reads_that_do_not_fit(reads):
    """Refused reads leave a context without reads, not one whose sizes are theirs and whose buffers are not."""
    few = reads[:5_000]
    with context(few, 32) as P:
        P.build_index()
        want = P.construct_string_graph()
        many = np.full((5_000_000, 100), 1, np.uint8)
        hog = fill(many.size // 2)
        with pytest.raises(pq.PQError) as refused:
            P.set_reads(many, T)
        assert refused.value.code == 3
        for call in (lambda: P.sort(0), P.build_index, lambda: P.build_fm(1), P.overlaps, P.counts, P.graph):
            with pytest.raises(pq.PQError) as state:
                call()
            assert state.value.code == 5
        del hog
        torch.cuda.empty_cache()
        P.construct_index(few, T)
        got = P.construct_string_graph()
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), getattr(want, f)), f
