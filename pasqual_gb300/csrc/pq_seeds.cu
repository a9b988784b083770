// pq_seeds.cu — the per-read seed intervals the reference's suffix sort records as a side effect
// (index_t.interval_start / interval_end / interval_depth; src/sufsort.c:178-209, 322-334),
// computed from a finished suffix array.
//
// The reference sorts each slot by counting passes on triplets at depths 3 and 6, then recurses
// from depth 9 (process_slot_1) three bases at a time; a bucket holding suffixes that share D
// bases is recursed into when it has more than one suffix, except that a bucket whose size times
// (L - D + 3) is below INSERT_SORT_SIZE (3500, src/common.h:57) is finished by insertion sort
// instead.  Whenever a bucket of depth D <= t is visited -- by the recursion or by the insertion
// sort -- every suffix in it that is exactly D bases long (the last D bases of its read) records
// the bucket as its read's seed, if D is deeper than the read's seed so far.  So read r's seed is
// the deepest such D together with the bucket's first row and size.
//
// Given the suffix array, bucket structure is a question of longest common prefixes: the rows of
// one depth-D bucket are a run of rows in which consecutive suffixes share at least D bases.  This
// file computes the common prefix of every pair of adjacent rows (capped at the deepest depth
// that matters, 3 * floor(t / 3)) and the minima of 64, 64^2 and 64^3 of them, by which a row's
// bucket at any depth is found in a few loads whatever its size.  A bucket at depth D is visited when
// all its ancestors were recursed into and it holds more than one suffix; it is recursed into itself
// when it was visited and (D == 9 or its size times (L - D + 3) is at least 3500, in the index
// width's unsigned arithmetic, as the reference's test wraps).  A suffix of exactly D bases is a
// prefix of all others of its bucket, so such suffixes are the bucket's first rows: only the rows
// that begin a bucket of their own length's depth are tested.  A read's deepest record wins.
//
// Buckets never span the reference's five sort slots (they share at least 3 bases), so running
// this over the rows of one slot gives exactly the records that slot's suf_sort call makes.
#include "pq_index.cuh"

namespace pq {

namespace {

constexpr idx_t kInsertSortSize = 3500;      // INSERT_SORT_SIZE

__device__ __forceinline__ uint64_t seed_window(const uint64_t* __restrict__ pk, size_t p) {
    const size_t w = p >> 5;
    const int s = int(p & 31) * 2;
    const uint64_t a = __ldg(pk + w), b = __ldg(pk + w + 1);
    return s ? ((a << s) | (b >> (64 - s))) : a;
}

// lcp[i - r0] = bases shared by the suffixes at rows i - 1 and i, at most `cap` (0 for i = r0).  Bound
// by the text windows' random sectors, one a row: a row's own, and its neighbour's by shuffle.
__global__ void k_seed_lcp(const idx_t* __restrict__ sa, const uint64_t* __restrict__ pk, DivL dl, size_t r0,
                           size_t r1, int cap, uint16_t* __restrict__ lcp) {
    const int lane = threadIdx.x & 31, L = int(dl.L);
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t w = r0 + (size_t(blockIdx.x) * blockDim.x + threadIdx.x) - lane; w < r1; w += stride) {
        const size_t i = w + lane;
        const idx_t q = i < r1 ? __ldg(sa + i) : 0;
        const uint64_t y = i < r1 ? seed_window(pk, size_t(q)) : 0;
        const int lq = L - int(q - idx_t(div_l(q, dl)) * idx_t(L));
        idx_t p = __shfl_up_sync(0xffffffffu, q, 1);
        uint64_t x = __shfl_up_sync(0xffffffffu, y, 1);
        int lp = __shfl_up_sync(0xffffffffu, lq, 1);
        if (i >= r1) continue;
        if (i == r0) {
            lcp[0] = 0;
            continue;
        }
        if (lane == 0) {
            p = __ldg(sa + i - 1);
            x = seed_window(pk, size_t(p));
            lp = L - int(p - idx_t(div_l(p, dl)) * idx_t(L));
        }
        int m = lp < lq ? lp : lq;
        m = m < cap ? m : cap;
        int c = 0;
        uint64_t d = x ^ y;
        while (!d) {
            c += 32;
            if (c >= m) break;
            d = seed_window(pk, size_t(p) + c) ^ seed_window(pk, size_t(q) + c);
        }
        if (d) c += __clzll((long long)d) >> 1;
        lcp[i - r0] = uint16_t(c < m ? c : m);
    }
}

// out[j] = minimum of in[64 j, 64 j + 64), as far as there are n
__global__ void k_min64(const uint16_t* __restrict__ in, size_t n, uint16_t* __restrict__ out) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    const size_t eights = (n + 63) / 64 * 8;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < (eights + 31) / 32 * 32; i += stride) {
        unsigned m = 0xffffffffu;
        if (8 * i + 8 <= n) {
            const uint4 v = reinterpret_cast<const uint4*>(in)[i];
            m = __vminu2(__vminu2(v.x, v.y), __vminu2(v.z, v.w));
        } else {
            for (size_t k = 8 * i; k < n; ++k) m = __vminu2(m, 0xffff0000u | in[k]);
        }
        m = min(m & 0xffffu, m >> 16);
        #pragma unroll
        for (int o = 1; o < 8; o <<= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
        if ((i & 7) == 0 && i < eights) out[i / 8] = uint16_t(m);
    }
}

constexpr int kSeedLevels = 4;
struct SeedRows {
    const uint16_t* lv[kSeedLevels];        // common prefixes, then minima of 64 of the level before
    size_t n[kSeedLevels];
};

// the first of lv[x, end) below D, or end
__device__ __forceinline__ size_t scan_up(const uint16_t* __restrict__ lv, size_t x, size_t end, unsigned D) {
    for (; x < end && (x & 7); ++x)
        if (lv[x] < D) return x;
    const unsigned dd = D | (D << 16);
    for (; x + 8 <= end; x += 8) {
        const uint4 v = *reinterpret_cast<const uint4*>(lv + x);
        if (__vcmpltu2(v.x, dd) | __vcmpltu2(v.y, dd) | __vcmpltu2(v.z, dd) | __vcmpltu2(v.w, dd)) break;
    }
    while (x < end && lv[x] >= D) ++x;
    return x;
}
// the first row >= x (of rows 0 ..) whose common prefix with the one before is below D, or their number
__device__ __forceinline__ size_t first_below(const SeedRows& R, size_t x, unsigned D) {
    int l = 0;
    while (true) {
        const size_t group = l == kSeedLevels - 1 ? R.n[l] : (x | 63) + 1;
        const size_t end = group < R.n[l] ? group : R.n[l];
        x = scan_up(R.lv[l], x, end, D);
        if (x < end) break;
        if (x >= R.n[l]) return R.n[0];
        x >>= 6;
        ++l;
    }
    while (l) {
        --l;
        x <<= 6;
        x = scan_up(R.lv[l], x, R.n[l], D);
    }
    return x;
}
// the last row <= x whose common prefix with the one before is below D (row 0's is 0)
__device__ __forceinline__ size_t last_below(const SeedRows& R, size_t x, unsigned D) {
    int l = 0;
    while (true) {
        const size_t begin = l == kSeedLevels - 1 ? 0 : x & ~size_t(63);
        while (x > begin && R.lv[l][x] >= D) --x;
        if (R.lv[l][x] < D) break;
        x = (begin >> 6) - 1;
        ++l;
    }
    while (l) {
        --l;
        x = x * 64 + 63;
        if (x >= R.n[l]) x = R.n[l] - 1;
        while (R.lv[l][x] >= D) --x;
    }
    return x;
}

// the depth a row's suffix (position p) can record, its length, or 0
__device__ __forceinline__ int record_depth(idx_t p, const DivL& dl, int dmax, idx_t& read) {
    read = idx_t(div_l(p, dl));
    const int len = int(dl.L) - int(p - read * idx_t(dl.L));
    return len >= 9 && len <= dmax && len % 3 == 0 ? len : 0;
}

// f(row, depth, read) for the rows that can record (one in six at L = 101, t = 63) and pass the test
// `first`, 32 of them a warp at a time: both follow dependent loads, and with a row a lane where it
// stands most lanes wait (2 M bases at 20x, both directions: 2.1 ms in the passes below, 1.4 with the
// queue).
constexpr int kSeedThreads = 256;
template <class First, class F>
__device__ __forceinline__ void for_record_rows(const idx_t* __restrict__ sa, size_t n, const DivL& dl, int dmax, First first, F f) {
    __shared__ size_t s_row[kSeedThreads / 32][64];
    __shared__ idx_t s_read[kSeedThreads / 32][64];
    __shared__ int s_depth[kSeedThreads / 32][64];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    int waiting = 0;
    for (size_t w = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) - lane; w < n; w += stride) {
        const size_t i = w + lane;
        idx_t read = 0;
        int D = i < n ? record_depth(__ldg(sa + i), dl, dmax, read) : 0;
        if (i < n && !first(i, D, read)) D = 0;
        const unsigned b = __ballot_sync(0xffffffffu, D != 0);
        if (D) {
            const int at = waiting + __popc(b & ((1u << lane) - 1u));
            s_row[wid][at] = i;
            s_read[wid][at] = read;
            s_depth[wid][at] = D;
        }
        waiting += __popc(b);
        __syncwarp();
        if (waiting >= 32) {
            waiting -= 32;
            f(s_row[wid][waiting + lane], s_depth[wid][waiting + lane], s_read[wid][waiting + lane]);
            __syncwarp();
        }
    }
    if (lane < waiting) f(s_row[wid][lane], s_depth[wid][lane], s_read[wid][lane]);
}

// visit[i] = 1 where row i begins a visited bucket at the depth of its own suffix's length.  With
// sizes that cannot wrap, the parent's test decides: its ancestors are larger and weigh more.
__global__ void __launch_bounds__(kSeedThreads) k_seed_visit(SeedRows R, const idx_t* __restrict__ sa, DivL dl, int dmax,
                                                             uint8_t* __restrict__ visit) {
    const size_t n = R.n[0];
    const uint16_t* const lcp = R.lv[0];
    const bool wraps = sizeof(idx_t) == 4 && (unsigned long long)n * dl.L > 0xffffffffull;
    for_record_rows(sa, n, dl, dmax,
        [&](size_t i, int D, idx_t) {
            const bool begins = D && lcp[i] < D && i + 1 < n && lcp[i + 1] >= D;
            visit[i] = begins && D <= 12;                   // depth 9's parent has no test, nor has 12's
            return begins && D > 12;
        },
        [&](size_t i, int D, idx_t) {
            bool ok = true;
            for (int d = D - 3; ok && d > 9; d -= 3) {
                const idx_t size = idx_t(first_below(R, i + 1, unsigned(d)) - last_below(R, i, unsigned(d)));
                ok = idx_t(size * idx_t(int(dl.L) - (d - 3))) >= kInsertSortSize;
                if (!wraps) break;
            }
            if (ok) visit[i] = 1;
        });
}

// the deepest record of every read that is deeper than its seed: won[read] (apply 0), then written
__global__ void __launch_bounds__(kSeedThreads) k_seed_record(SeedRows R, const idx_t* __restrict__ sa, DivL dl, int dmax,
                                                              const uint8_t* __restrict__ visit, size_t r0, int apply,
                                                              unsigned* __restrict__ won, uint16_t* __restrict__ depth,
                                                              idx_t* __restrict__ start, idx_t* __restrict__ size) {
    for_record_rows(sa, R.n[0], dl, dmax,
        [&](size_t, int D, idx_t read) { return D && (apply ? won[read] == unsigned(D) : depth[read] < D); },
        [&](size_t i, int D, idx_t read) {
            const size_t head = last_below(R, i, unsigned(D));
            if (!visit[head]) return;
            if (!apply) {
                atomicMax(won + read, unsigned(D));
            } else {
                depth[read] = uint16_t(D);
                start[read] = idx_t(r0 + head);
                size[read] = idx_t(first_below(R, i + 1, unsigned(D)) - head);
            }
        });
}

// the seed every read starts from in build_idx (src/index.c:495-502, 548-555): the interval of its
// last base (forward) or first base (backward) by C[], depth 1
struct SeedC {
    idx_t c[6];
};
__global__ void k_seed_init(const uint8_t* __restrict__ reads, idx_t num_reads, idx_t L, int dir, SeedC C,
                            uint16_t* __restrict__ depth, idx_t* __restrict__ start, idx_t* __restrict__ size) {
    for (size_t r = size_t(blockIdx.x) * blockDim.x + threadIdx.x; r < size_t(num_reads);
         r += size_t(gridDim.x) * blockDim.x) {
        const int ch = reads[r * size_t(L) + (dir ? 0 : size_t(L) - 1)];
        start[r] = C.c[ch];
        size[r] = C.c[ch + 1] - C.c[ch];
        depth[r] = 1;
    }
}

int grid_for_rows(size_t n, int per_block) {
    size_t g = (n + per_block - 1) / per_block;
    if (g > 152 * 64) g = 152 * 64;
    return int(g ? g : 1);
}

}  // namespace

cudaError_t seed_init(const uint8_t* reads, idx_t num_reads, idx_t L, int dir, const idx_t C[6], uint16_t* depth,
                      idx_t* start, idx_t* size, cudaStream_t st) {
    if (!num_reads) return cudaSuccess;
    SeedC c;
    for (int i = 0; i < 6; ++i) c.c[i] = C[i];
    k_seed_init<<<grid_for_rows(num_reads, 256), 256, 0, st>>>(reads, num_reads, L, dir, c, depth, start, size);
    note_launch();
    return cudaGetLastError();
}

static size_t seed_layout(size_t rows, size_t num_reads, size_t (&o)[kSeedLevels + 2], size_t (&n)[kSeedLevels]) {
    size_t used = 0, m = rows;
    auto take = [&](size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) & ~size_t(255);
        return at;
    };
    for (int l = 0; l < kSeedLevels; ++l, m = (m + 63) / 64) {
        n[l] = m;
        o[l] = take(m * sizeof(uint16_t));
    }
    o[kSeedLevels] = take(rows);
    o[kSeedLevels + 1] = take(num_reads * sizeof(unsigned));
    return used;
}

size_t sort_seeds_tmp_bytes(size_t rows, size_t num_reads) {
    size_t o[kSeedLevels + 2], n[kSeedLevels];
    return seed_layout(rows, num_reads, o, n);
}

// Three passes over the rows and one over their text.  2 M bases at 20x, both directions, 80 M rows:
// 6.2 ms with a pass per depth over all rows whose ancestors were recursed into, now 2.2, of which 0.7
// for the text, 0.7 for the visits and 0.8 for the records.
cudaError_t sort_seeds(const idx_t* sa, const uint64_t* pk, idx_t num_reads, idx_t L, int t, size_t r0, size_t r1,
                       uint16_t* depth, idx_t* start, idx_t* size, void* tmp, size_t tmp_bytes, cudaStream_t st) {
    if (r1 <= r0 || t < 9) return cudaSuccess;
    const size_t rows = r1 - r0;
    size_t o[kSeedLevels + 2];
    SeedRows R;
    if (tmp_bytes < seed_layout(rows, size_t(num_reads), o, R.n)) return cudaErrorInvalidValue;
    char* p = static_cast<char*>(tmp);
    const DivL dl = make_divl(uint32_t(L));
    const int dmax = 3 * (t / 3), grid = grid_for_rows(rows, 256);
    uint16_t* lv[kSeedLevels];
    for (int l = 0; l < kSeedLevels; ++l) R.lv[l] = lv[l] = reinterpret_cast<uint16_t*>(p + o[l]);
    uint8_t* visit = reinterpret_cast<uint8_t*>(p + o[kSeedLevels]);
    unsigned* won = reinterpret_cast<unsigned*>(p + o[kSeedLevels + 1]);
    cudaError_t e = cudaMemsetAsync(won, 0, size_t(num_reads) * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    k_seed_lcp<<<grid, 256, 0, st>>>(sa, pk, dl, r0, r1, dmax, lv[0]);
    note_launch();
    for (int l = 1; l < kSeedLevels; ++l) {
        k_min64<<<grid_for_rows((R.n[l - 1] + 7) / 8, 256), 256, 0, st>>>(lv[l - 1], R.n[l - 1], lv[l]);
        note_launch();
    }
    k_seed_visit<<<grid, kSeedThreads, 0, st>>>(R, sa + r0, dl, dmax, visit);
    note_launch();
    for (int apply = 0; apply < 2; ++apply) {
        k_seed_record<<<grid, kSeedThreads, 0, st>>>(R, sa + r0, dl, dmax, visit, r0, apply, won, depth, start, size);
        note_launch();
    }
    return cudaGetLastError();
}

}  // namespace pq
