"""The work whose time and results are followed: whole assemblies from host reads, overlap searches
on a resident index, suffix sorts in caller-owned device memory, and the index handed to the
reference's own structures, over the read lengths, overlaps, index widths and search options of
this repository's workloads (pasqual_gb300/synth.py), golden cases and benchmark.

A case names a genome shape (size, GC, repeats and their divergence, dinucleotide runs) and a read
set drawn from it (length L, coverage, error rate), as pasqual_gb300.synth draws them; the same
sampling is done here on the GPU, since read sets of a gigabyte take numpy many seconds.
"""
import ctypes as ct
import math
import random

import numpy as np
import torch

import pasqual_gb300 as pq

STATIC_MAX = 1 << 20            # suffixes pq_suffix_sort_static accepts


def _case(name, kind, **kw):
    c = {"name": name, "kind": kind, "width": 32, "genome": 20_000, "gc": 0.41, "repeat": 0.1, "div_lo": 0.01,
         "div_hi": 0.01, "runs": 0.0, "L": 100, "cov": 20.0, "err": 0.005, "t": 63, "mode": 1, "chunk": 0,
         "locked": True, "dir": 0}
    c.update(kw)
    return c


def listed():
    return [
        # A latency-bound caller's sort: the reads of one locus, in its own device buffers.
        _case("static_50k", "static", genome=2_000, cov=25.0),
        # The largest sort that entry point takes, 64-bit index, reversed reads, odd count.
        _case("static_1M_u64", "static", width=64, genome=52_100, L=150, cov=20.0, err=0.003, dir=1),
        # A plasmid or an amplicon: the whole call on 4 K reads from pageable memory, where
        # launches, copies and synchronisations count (the build's own smoke workload).
        _case("assemble_20k", "assemble", gc=0.45, err=0.003, locked=False),
        # A bacterial genome in short error-free reads, 40x (the 1 Mbp workload).
        _case("assemble_1M_L50", "assemble", genome=1_000_000, gc=0.5, repeat=0.0, L=50, cov=40.0, err=0.0, t=31,
              locked=False),
        # The index as the reference's own program receives it: both FM-indexes exported in its
        # layout with the seed intervals its sort records, for reads of odd length.
        _case("index_2M_L101", "index", genome=2_000_000, L=101, cov=25.0, t=47, locked=False),
        # The 50 Mbp, 100 bp, 30x workload at 1/10 genome: an ordinary assembly.
        _case("assemble_5M_L100", "assemble", genome=5_000_000, cov=30.0),
        # Long reads with a long minimum overlap, odd length: many words per comparison.
        _case("assemble_10M_L233", "assemble", genome=10_000_000, gc=0.45, repeat=0.08, L=233, cov=20.0, t=95),
        # The largest: the 250 Mbp workload's shape at 1/4 genome, 64-bit index of 1.2 G suffixes,
        # sorted in chunks a quarter of the default's, so in as many chunks as the full workload.
        _case("assemble_62M_u64_chunked", "assemble", width=64, genome=62_500_000, gc=0.42, repeat=0.15,
              div_lo=0.005, div_hi=0.02, t=55, chunk=1 << 28),
        # The benchmark's own step: a search over every read with both indexes resident, the
        # 250 Mbp workload's shape at 1/8 genome.
        _case("search_31M_u64", "search", width=64, genome=31_250_000, gc=0.42, repeat=0.15, div_lo=0.005,
              div_hi=0.02, t=55),
        # The same step by the reference's method (seed mode 0: backward search and the DFS).
        _case("search_walk_5M", "search", genome=5_000_000, cov=30.0, mode=0),
        # Low-complexity sequence: the 200 Mbp workload with 2 % dinucleotide runs at 1/100 genome,
        # whose run reads have thousands of candidates a side.
        _case("search_runs_2M_u64", "search", width=64, genome=2_000_000, gc=0.40, repeat=0.12, runs=0.02, L=150,
              err=0.003),
        # Read sets of uneven length and mixed minimum overlap in one queued, graph-replayed launch
        # with learned-index windows (the 100 Mbp queued workload at 1/10 genome, seven sets).
        _case("queue_10M_mixed", "queue", genome=10_000_000, gc=0.45, repeat=0.08, cov=22.0, mode=2,
              Ls="232,228,127,216,122,202,148", ts="63,95,63,31,63,31,47"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["static", "static", "assemble", "assemble", "assemble", "search", "search", "index", "queue"])
    L = rng.randint(40, 250)
    c = _case("", kind, width=rng.choice([32, 64]), gc=round(rng.uniform(0.38, 0.52), 3),
              repeat=round(rng.choice([0.0, rng.uniform(0.05, 0.15)]), 3), div_hi=round(rng.uniform(0.01, 0.02), 4),
              L=L, cov=round(rng.uniform(15, 40), 1), err=round(rng.choice([0.0, rng.uniform(0.002, 0.008)]), 4),
              t=rng.randint(31, min(L - 5, 120)), locked=rng.random() < 0.5, dir=rng.randint(0, 1))
    del c["name"]
    if kind == "static":
        c["genome"] = max(4 * L, int(log(20_000, STATIC_MAX) / c["cov"]))
    elif kind == "queue":
        sets = rng.randint(2, 7)
        Ls = [rng.randint(75, 250) for _ in range(sets)]
        c.update(genome=log(50_000, 8_000_000), cov=25.0, mode=rng.choice([1, 2]), Ls=",".join(map(str, Ls)),
                 ts=",".join(str(rng.choice([x for x in (31, 47, 63, 95) if x < n - 4])) for n in Ls))
    else:
        c["genome"] = log(20_000, 10_000_000 if kind != "index" else 3_000_000)
        if kind == "search":
            c["mode"] = rng.choice([0, 1, 1, 2])
        if kind != "index" and c["mode"] == 1 and rng.random() < 0.25:
            c.update(runs=0.02, genome=min(c["genome"], 1_500_000), cov=min(c["cov"], 20.0))
        if kind == "assemble" and c["genome"] > 1_000_000 and rng.random() < 0.4:
            c["chunk"] = max(1 << 22, int(c["genome"] * c["cov"] / rng.randint(2, 6)))
    return c


# ------------------------------------------------------------------------------------- inputs

def _genome(c, g, host):
    """Base codes 0..3 on the GPU: i.i.d. bases, then 1-5 kbp copies at the case's divergence,
    then dinucleotide runs of 20-200 bp."""
    n, gc = c["genome"], c["gc"]
    u = torch.rand(n, generator=g, device="cuda")
    s = ((u > (1 - gc) / 2).to(torch.uint8) + (u > 0.5) + (u > (1 + gc) / 2)).to(torch.uint8)
    done = 0
    while done < int(c["repeat"] * n) and n > 6000:
        m = host.randint(1000, 5000)
        a, b = host.randrange(n - m), host.randrange(n - m)
        seg = s[a:a + m].clone()
        mut = torch.rand(m, generator=g, device="cuda") < host.uniform(c["div_lo"], c["div_hi"])
        seg = torch.where(mut, (seg + torch.randint(1, 4, (m,), generator=g, device="cuda", dtype=torch.uint8)) % 4, seg)
        s[b:b + m] = seg
        done += m
    done = 0
    while done < int(c["runs"] * n) and n > 400:
        m = host.randint(20, 200)
        at = host.randrange(n - m)
        a, b = host.sample(range(4), 2)
        s[at:at + m:2] = a
        s[at + 1:at + m:2] = b
        done += m
    return s


def _dedup(rd):
    """The first read of every group of equal or reverse-complement reads, in order."""
    nr, L = rd.shape
    keys = []
    for cols, flip in ((range(L), 0), (range(L - 1, -1, -1), 3)):
        h = torch.full((nr,), 0x1234567, dtype=torch.int64, device="cuda")
        for j in cols:
            h = h * 0x5851F42D4C957F2D + (rd[:, j] ^ flip)
            if j % 8 == 0:
                h ^= (h >> 29) & 0x7FFFFFFFF
        keys.append(h)
    key, order = torch.sort(torch.minimum(*keys), stable=True)
    first = torch.ones(nr, dtype=torch.bool, device="cuda")
    first[1:] = key[1:] != key[:-1]
    keep = torch.zeros(nr, dtype=torch.bool, device="cuda")
    keep[order[first]] = True
    return rd[keep]


def _kept(genome, cov, L):
    """Reads of a set: a little under the number of different starts that sampling at `cov` gives,
    the same for every seed."""
    return max(4, int(0.95 * genome * (1 - math.exp(-cov / L))))


def _reads(c, s, g, L, cov):
    """A read set (codes 1..4) on the GPU: sampled at `cov`, duplicates dropped, cut to the same
    number of reads for every seed."""
    want = _kept(s.numel(), cov, L)
    rd = _dedup(_sample(c, s, g, L, max(int(s.numel() * cov // L), 4)))
    while rd.shape[0] < want:
        rd = _dedup(torch.cat([rd, _sample(c, s, g, L, want - rd.shape[0] + want // 16 + 16)]))
    return rd[:want] + 1


def _sample(c, s, g, L, nr):
    """Reads (codes 0..3): uniform starts, half of them reverse complements, substitution errors."""
    n = s.numel()
    out = torch.empty((nr, L), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 26) // L)
    at = torch.arange(L, device="cuda")
    for i in range(0, nr, step):
        m = min(step, nr - i)
        start = torch.randint(0, n - L + 1, (m,), generator=g, device="cuda")
        rc = torch.rand(m, generator=g, device="cuda") < 0.5
        blk = s[start[:, None] + torch.where(rc[:, None], L - 1 - at, at)]
        blk = torch.where(rc[:, None], 3 - blk, blk)
        if c["err"] > 0:
            e = torch.rand((m, L), generator=g, device="cuda")
            # 0 < e / err < 1 spreads evenly over the three other bases
            blk = torch.where(e < c["err"], (blk + 1 + (e * (3 / c["err"])).clamp(max=2.5).to(torch.uint8)) % 4, blk)
        out[i:i + m] = blk
    return out


def _host(rd, locked, width):
    a = pq.host_empty(tuple(rd.shape), np.uint8, width) if locked else np.empty(tuple(rd.shape), np.uint8)
    torch.from_numpy(a).copy_(rd)
    return a


def _room(c, nr):
    """A Graph whose arrays hold the result (the caller's buffers, kept from call to call), in
    page-locked memory when the reads are; zero past the edges there are."""
    w = c["width"]
    # errors leave reads that no other read's overlap covers, run reads overlap each other
    per = 3 if c["err"] * c["L"] <= 0.5 and c["cov"] <= 30 else 6 + int(2 * c["cov"] * min(1.0, c["err"] * c["L"]))
    ne = (per + (96 if c["runs"] else 0)) * nr + 4096
    idx = np.uint64 if w == 64 else np.uint32

    def e(n, dt):
        a = pq.host_empty((n,), dt, w) if c["locked"] else np.empty(n, dt)
        a[:] = 0
        return a

    return pq.Graph(num_B=e(nr, np.uint16), num_F=e(nr, np.uint16), olp_B=e(nr, np.int32), olp_F=e(nr, np.int32),
                    edge_off=e(nr + 1, np.uint64), dest=e(ne, idx), length=e(ne, np.uint16), etype=e(ne, np.uint8),
                    trans=e(ne, np.int32))


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)
    host = random.Random(seed)
    s = _genome(c, g, host)
    st = {"case": c}
    if c["kind"] == "queue":
        Ls, ts = ([int(x) for x in c[k].split(",")] for k in ("Ls", "ts"))
        st["ctx"], st["out"] = [], []
        for L, t in zip(Ls, ts):
            c = dict(case, L=L, cov=case["cov"] / len(Ls))
            rd = _host(_reads(c, s, g, L, c["cov"]), c["locked"], c["width"])
            P = pq.Pasqual(c["width"])
            P.set_seed_mode(c["mode"])
            P.construct_index(rd, t)
            P.overlaps()            # each set's own search, which also trains its learned index
            st["ctx"].append(P)
            st["out"].append(_room(c, rd.shape[0]))
    else:
        rd = _reads(c, s, g, c["L"], c["cov"])
        if c["kind"] == "static":
            rd = rd[:STATIC_MAX // c["L"]].contiguous()
            st["reads"] = rd
            st["sa"] = torch.empty(rd.numel(), dtype=torch.int64 if c["width"] == 64 else torch.int32, device="cuda")
            st["sort"] = f = pq.load_library(c["width"]).pq_suffix_sort_static
            f.restype = ct.c_int
            f.argtypes = [ct.c_void_p, ct.c_uint64 if c["width"] == 64 else ct.c_uint32, ct.c_int, ct.c_int,
                          ct.c_void_p, ct.c_void_p]
        else:
            st["reads"] = _host(rd, c["locked"], c["width"])
            st["ctx"] = P = pq.Pasqual(c["width"])
            P.set_seed_mode(c["mode"])
            P.set_sort_chunk(c["chunk"])
            if c["kind"] != "index":
                st["out"] = _room(c, rd.shape[0])
            if c["kind"] == "search":
                P.construct_index(st["reads"], c["t"])
    del s, rd
    torch.cuda.empty_cache()        # the library allocates its own device memory
    return st


# ---------------------------------------------------------------------------------------- a pass

def _signed(a):
    """The same bytes as signed integers (torch has few operations on unsigned ones)."""
    return a.view("i%d" % a.dtype.itemsize) if a.dtype.itemsize > 1 else a


def _graph(P, out):
    """The graph, read into the caller's buffers: those, whole."""
    gr = P.graph(out)
    full = out if len(gr.dest) <= len(out.dest) else gr
    return [_signed(a) for a in (full.num_B, full.num_F, full.olp_B, full.olp_F, full.edge_off, full.dest, full.length,
                                 full.etype, full.trans)]


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "static":
        rd, sa = state["reads"], state["sa"]
        rc = state["sort"](rd.data_ptr(), rd.shape[0], rd.shape[1], c["dir"], sa.data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        if rc:
            raise pq.PQError(rc, "pq_suffix_sort_static")
        return sa
    if kind == "queue":
        pq.overlaps_batched(state["ctx"], graph=True)
        return [_graph(P, out) for P, out in zip(state["ctx"], state["out"])]
    P = state["ctx"]
    if kind == "search":
        P.overlaps()
        return _graph(P, state["out"])
    P.construct_index(state["reads"], c["t"])
    if kind == "assemble":
        P.overlaps()
        return _graph(P, state["out"])
    return [[_signed(a) for a in P.index_ref(d) + P.sort_seeds(d)] for d in (0, 1)]


def work(case):
    """Bytes a pass cannot do without: the reads in, or the packed texts and suffix arrays of a
    resident index where the case starts from one; the suffix array, index or graph out (about two
    edges a read).  The path compares and counts: no floating-point operations to speak of."""
    c = case
    idx = c["width"] // 8
    if c["kind"] == "queue":
        Ls = [int(x) for x in c["Ls"].split(",")]
        sets = [(_kept(c["genome"], c["cov"] / len(Ls), L), L) for L in Ls]
    else:
        sets = [(_kept(c["genome"], c["cov"], c["L"]), c["L"])]
    total = 0.0
    for nr, L in sets:
        n = nr * L
        if c["kind"] == "static":
            n = min(n, STATIC_MAX)
        graph = nr * (2 + 2 + 4 + 4 + 8) + 2 * nr * (idx + 7)
        total += {"static": n + n * idx, "assemble": n + graph, "index": n + 2 * (n / 64 * (5 * 8 + 5 * idx) + nr * (3 * idx + 2)),
                  "search": 2 * (n / 4 + n * idx) + graph, "queue": 2 * (n / 4 + n * idx) + graph}[c["kind"]]
    return {"bytes": total, "flops": 0.0}


def exact(case, seed):
    """Every output is a suffix position, a row, a read id, a length or a count: whole numbers, for
    which equality is asked.  None is a rounded value."""
    return None
