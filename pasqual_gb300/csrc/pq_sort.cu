// pq_sort.cu — suffix sort of the reads (forward) or of the reversed reads (backward).
//
// Replaces transform_to_triplet[_reverse], initial_sort and suf_sort (src/sufsort.c:80-614) as
// driven by build_idx (src/index.c:558-585).  The reference sorts in 5 slots by an MSD counting
// sort on 3-character "triplet" ranks with insertion sort for small buckets; its single-threaded
// output order is: read-bounded suffix strings, end-of-read lowest, ties by text position.
//
// GB300 design: the text is packed 2 bits per base.  Every suffix becomes one 64-bit element --
// its next bases, min(length, head), its position and its BWT symbol, highest first -- made
// straight from the text by the first of two partition passes on the leading bases (most
// significant digit first).  Elements are distinct and carry their position, so the partitions
// need not be stable: a tile reserves its place in every bucket with one atomic per bucket, and
// there is no per-tile count matrix, no scan of one and no second sweep.  The buckets (about a
// thousand suffixes) are then finished one per CTA in shared memory: split once more by their
// next differing bits, every sub-bucket of up to 32 suffixes sorted by one warp on the rest of its
// bases, and the finished rows streamed out with their BWT symbols and k-mer table entries.
// Suffixes of a few bases, of which every string has nr / 4^m equal copies, are sorted apart by a
// stable radix sort.  Buckets too large for shared memory (low-complexity sequence) are split
// further by the host, by the highest bits in which their elements differ; groups of more than a
// thousand suffixes equal in all bases of their elements get new elements of their next bases.
// Reads longer than the shared-memory network's words are sorted by prefix doubling on 29-base
// 64-bit keys: ranks by (rank(p), rank(p+h) or "empty" past the read end) for h = 29, 58, 116, ...
#include "pq_sort.cuh"
#include "pq_index.cuh"
#include "pq_pack.h"
#include "pq_ranges.h"

#include <algorithm>
#include <vector>

namespace pq {

constexpr int kWide = 29;                 // bases per 64-bit key of the prefix doubling

__host__ __device__ __forceinline__ size_t zmin(size_t a, size_t b) { return a < b ? a : b; }

static inline unsigned grid_for(size_t work, int threads, int per_sm = 8) {
    size_t g = (work + threads - 1) / threads;
    size_t cap = size_t(152) * per_sm * 4;
    return unsigned(std::max<size_t>(1, std::min(g, cap)));
}

static int device_sms() {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// ------------------------------------------------------------------------------ packed text

// 32 bases per word, first base in the top two bits (A=0 .. T=3).  The forward text of a whole
// word comes in two 16-byte loads; the backward text in steps of eight bases with one division for
// the first (the read offset then steps and wraps).
__device__ __forceinline__ uint64_t swap8(uint32_t lo, uint32_t hi) {
    return (uint64_t(__byte_perm(lo, 0, 0x0123)) << 32) | __byte_perm(hi, 0, 0x0123);
}
// Bound by the bytes read (1.13 G bases, both directions: 0.70 ms, 1.43 a base at a time).  No byte outside
// the reads is read: at their ends, where the words of eight would hold others, a base at a time.
__global__ void k_pack_text(const uint8_t* __restrict__ reads, size_t n, DivL dl, int dir, size_t nwords,
                            uint64_t* __restrict__ pk) {
    const size_t stride = size_t(gridDim.x) * blockDim.x, L = dl.L;
    const bool vec = dir == 0 && reinterpret_cast<uintptr_t>(reads) % 16 == 0;
    for (size_t w = size_t(blockIdx.x) * blockDim.x + threadIdx.x; w < nwords; w += stride) {
        const size_t p0 = w * 32;
        uint64_t v = 0;
        if (vec && p0 + 32 <= n) {
            const uint4 a = *reinterpret_cast<const uint4*>(reads + p0);
            const uint4 b = *reinterpret_cast<const uint4*>(reads + p0 + 16);
            v = (uint64_t(pack8(swap8(a.x, a.y))) << 48) | (uint64_t(pack8(swap8(a.z, a.w))) << 32) |
                (uint64_t(pack8(swap8(b.x, b.y))) << 16) | pack8(swap8(b.z, b.w));
        } else if (p0 < n) {
            size_t r = L == 1 ? p0 : size_t(div_l(p0, dl)), off = p0 - r * L;
            if (dir == 1 && L >= 8 && pack_inside(reinterpret_cast<uintptr_t>(reads), n, p0, L)) {
                v = pack_backward(reinterpret_cast<uintptr_t>(reads), r, off, L,
                                  [](uintptr_t a) { return *reinterpret_cast<const uint64_t*>(a); });
            } else {
                for (int j = 0; j < 32; ++j) {
                    const size_t p = p0 + size_t(j);
                    uint64_t c = 0;
                    if (p < n) c = uint64_t((dir == 0 ? reads[p] : reads[r * L + (L - 1 - off)]) - 1);
                    v = (v << 2) | c;
                    if (++off == L) {
                        off = 0;
                        ++r;
                    }
                }
            }
        }
        pk[w] = v;
    }
}

__device__ __forceinline__ uint64_t window(const uint64_t* __restrict__ pk, size_t p) {
    size_t w = p >> 5;
    int s = int(p & 31) * 2;
    uint64_t a = pk[w];
    uint64_t b = pk[w + 1];
    return s ? ((a << s) | (b >> (64 - s))) : a;
}

// the 64-bit key of a suffix whose bases start the window x and of which m exist (m >= 0): 29 bases
// (padded with A, first base highest) in bits 63..6, how many of them exist (0..29) in bits 5..0
__device__ __forceinline__ uint64_t make_wide_key(uint64_t x, int m) {
    const int w = m < kWide ? m : kWide;
    if (w <= 0) return 0;
    return (x & (~uint64_t(0) << (64 - 2 * w))) | uint64_t(w);
}

__global__ void k_init_keys(const uint64_t* __restrict__ pk, size_t n, idx_t L, uint64_t* __restrict__ key,
                            idx_t* __restrict__ val) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t p = size_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += stride) {
        key[p] = make_wide_key(window(pk, p), int(L - idx_t(p % L)));
        val[p] = idx_t(p);
    }
}

// ------------------------------------------------------------------------------ radix sort

constexpr int RS_THREADS = 256;
constexpr int RS_IPT = 8;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_MAX_CTAS = 152 * 4;

// Digit histograms of all byte positions over the whole key array (order independent): a pass
// whose digit is constant over all keys is the identity and is skipped.
template <class K>
__global__ void k_digit_hist(const K* __restrict__ key, size_t n, unsigned long long* __restrict__ hist) {
    constexpr int D = int(sizeof(K));
    __shared__ unsigned int h[D][256];
    for (int i = threadIdx.x; i < D * 256; i += blockDim.x) (&h[0][0])[i] = 0;
    __syncthreads();
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        const K k = key[i];
        #pragma unroll
        for (int d = 0; d < D; ++d) atomicAdd(&h[d][(k >> (8 * d)) & 255], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < D * 256; i += blockDim.x)
        if ((&h[0][0])[i]) atomicAdd(&hist[i], (unsigned long long)(&h[0][0])[i]);
}

template <class K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_upsweep(const K* __restrict__ key, size_t n, int shift,
                                                           size_t part, unsigned long long* __restrict__ cnt) {
    __shared__ unsigned int h[RS_WARPS][256];
    const int warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < RS_WARPS * 256; i += RS_THREADS) (&h[0][0])[i] = 0;
    __syncthreads();
    const size_t beg = size_t(blockIdx.x) * part;
    const size_t end = zmin(n, beg + part);
    for (size_t i = beg + threadIdx.x; i < end; i += RS_THREADS)
        atomicAdd(&h[warp][(key[i] >> shift) & 255], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += RS_THREADS) {
        unsigned long long s = 0;
        #pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) s += h[w][d];
        cnt[size_t(d) * gridDim.x + blockIdx.x] = s;
    }
}

// one CTA per digit: exclusive scan of the digit's counts over the parts, in place, and their total
__global__ void __launch_bounds__(RS_THREADS) k_rs_scan(unsigned long long* __restrict__ cnt, unsigned ctas,
                                                        unsigned long long* __restrict__ total) {
    __shared__ unsigned long long wsum[RS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned long long* row = cnt + size_t(blockIdx.x) * ctas;
    unsigned long long carry = 0;
    for (unsigned b = 0; b < ctas; b += RS_THREADS) {
        const unsigned i = b + tid;
        const unsigned long long v = i < ctas ? row[i] : 0ull;
        unsigned long long x = v;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        unsigned long long pre = carry, all = 0;
        #pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            pre += w < warp ? wsum[w] : 0ull;
            all += wsum[w];
        }
        if (i < ctas) row[i] = pre + x - v;
        carry += all;
        __syncthreads();
    }
    if (tid == 0) total[blockIdx.x] = carry;
}

// 16-byte asynchronous global -> shared copies (bypassing registers and L1)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = unsigned(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Downsweep configuration: 512 threads (tiles of 4096) for 32-bit keys and values, whose tile,
// staging buffer and reorder buffer fit two CTAs per SM; 256 threads otherwise.
template <class K, class V>
struct RsCfg {
    static constexpr int threads = (sizeof(K) == 4 && sizeof(V) == 4) ? 512 : 256;
    static constexpr int tile = threads * RS_IPT;
    static constexpr int min_blocks = threads == 512 ? 2 : (sizeof(K) == 4 ? 4 : 3);   // CTAs per SM
};
constexpr int RS_TILE_MAX = 4096;           // parts are whole multiples of every tile size

// One CTA per contiguous part of the input, tiles in order.  Per tile: every thread takes its
// RS_IPT (key, value) pairs, from the staging buffer when the tile was prefetched there (whole,
// 16-byte aligned tiles: the next tile's copy runs while this one is ranked and written), else
// straight from global memory; each warp ranks its rows by digit (8 ballots per row give the lanes
// with the same digit; a per-warp count per digit in shared memory carries the rank from row to
// row), the tile is reordered by digit in shared memory and written out in runs per digit at the
// part's running digit offsets.
template <class K, class V>
__global__ void __launch_bounds__(RsCfg<K, V>::threads, RsCfg<K, V>::min_blocks)
k_rs_downsweep(const K* __restrict__ kin, const V* __restrict__ vin, K* __restrict__ kout, V* __restrict__ vout,
               size_t n, int shift, size_t part, const unsigned long long* __restrict__ offs,
               const unsigned long long* __restrict__ total, int staged) {
    constexpr int T = RsCfg<K, V>::threads;
    constexpr int TILE = RsCfg<K, V>::tile;
    constexpr int NW = T / 32;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    K* stk = reinterpret_cast<K*>(rs_smem);                          // staging: keys, values
    V* stv = reinterpret_cast<V*>(stk + TILE);
    K* sk = reinterpret_cast<K*>(stv + TILE);                         // reorder buffer
    V* sv = reinterpret_cast<V*>(sk + TILE);
    unsigned (*wcnt)[256] = reinterpret_cast<unsigned (*)[256]>(sv + TILE);
    unsigned* tcount = &wcnt[NW][0];
    unsigned* dstart = tcount + 256;
    unsigned* wtot = dstart + 256;
    unsigned long long* base = reinterpret_cast<unsigned long long*>(wtot + 32);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1;
    {   // a digit's place: the totals of the smaller digits plus the earlier parts' counts
        __shared__ unsigned long long s_tot[8];
        unsigned long long v0 = 0, x = 0;
        if (tid < 256) {
            v0 = total[tid];
            x = v0;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_tot[warp] = x;
        }
        __syncthreads();
        if (tid < 256) {
            for (int w = 0; w < warp; ++w) x += s_tot[w];
            base[tid] = x - v0 + offs[size_t(tid) * gridDim.x + blockIdx.x];
        }
    }
    const size_t beg = size_t(blockIdx.x) * part;
    const size_t end = zmin(n, beg + part);
    auto prefetch = [&](size_t t) {
        constexpr int KC = TILE * int(sizeof(K)) / 16, VC = TILE * int(sizeof(V)) / 16;
        for (int i = tid; i < KC; i += T)
            cp_async16(reinterpret_cast<char*>(stk) + 16 * i, reinterpret_cast<const char*>(kin + t) + 16 * size_t(i));
        for (int i = tid; i < VC; i += T)
            cp_async16(reinterpret_cast<char*>(stv) + 16 * i, reinterpret_cast<const char*>(vin + t) + 16 * size_t(i));
        cp_async_commit();
    };
    if (staged && beg + TILE <= end) prefetch(beg);
    for (size_t t0 = beg; t0 < end; t0 += TILE) {
        for (int i = lane; i < 256; i += 32) wcnt[warp][i] = 0;
        K k[RS_IPT];
        V v[RS_IPT];
        unsigned int lr[RS_IPT];
        const int j0 = warp * 32 * RS_IPT + lane;
        const size_t row0 = t0 + j0;
        if (staged && t0 + TILE <= end) {
            cp_async_wait_all();
            __syncthreads();
            #pragma unroll
            for (int r = 0; r < RS_IPT; ++r) {
                k[r] = stk[j0 + r * 32];
                v[r] = stv[j0 + r * 32];
            }
            __syncthreads();                                    // the staging buffer is free again
            if (t0 + 2 * size_t(TILE) <= end) prefetch(t0 + TILE);
        } else {
            #pragma unroll
            for (int r = 0; r < RS_IPT; ++r) {
                const size_t idx = row0 + r * 32;
                k[r] = idx < end ? kin[idx] : K(0);
                v[r] = idx < end ? vin[idx] : V(0);
            }
            __syncwarp();
        }
        #pragma unroll
        for (int r = 0; r < RS_IPT; ++r) {
            const bool valid = row0 + r * 32 < end;
            const int d = valid ? int((k[r] >> shift) & 255) : -1;
            unsigned peers = __ballot_sync(0xffffffffu, valid);
            #pragma unroll
            for (int b = 0; b < 8; ++b) {
                unsigned bits = __ballot_sync(0xffffffffu, (d >> b) & 1);
                peers &= ((d >> b) & 1) ? bits : ~bits;
            }
            unsigned before = 0;
            if (valid) before = wcnt[warp][d];
            __syncwarp();
            if (valid && (peers & lt_mask) == 0) wcnt[warp][d] = before + __popc(peers);
            __syncwarp();
            lr[r] = before + __popc(peers & lt_mask);
        }
        __syncthreads();
        // per digit: warp prefixes and tile count
        for (int d = tid; d < 256; d += T) {
            unsigned run = 0;
            #pragma unroll
            for (int w = 0; w < NW; ++w) {
                unsigned c = wcnt[w][d];
                wcnt[w][d] = run;
                run += c;
            }
            tcount[d] = run;
        }
        __syncthreads();
        // exclusive scan of tcount over the 256 digits (one per thread of the first 8 warps)
        {
            unsigned v0 = 0, x = 0;
            if (tid < 256) {
                v0 = tcount[tid];
                x = v0;
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    unsigned y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == 31) wtot[warp] = x;
            }
            __syncthreads();
            if (tid < 256) {
                unsigned pre = 0;
                for (int w = 0; w < warp; ++w) pre += wtot[w];
                dstart[tid] = pre + x - v0;
            }
        }
        __syncthreads();
        #pragma unroll
        for (int r = 0; r < RS_IPT; ++r) {
            if (row0 + r * 32 < end) {
                const int d = int((k[r] >> shift) & 255);
                const unsigned pos = dstart[d] + wcnt[warp][d] + lr[r];
                sk[pos] = k[r];
                sv[pos] = v[r];
            }
        }
        __syncthreads();
        const int cnt = int(zmin(size_t(TILE), end - t0));
        for (int j = tid; j < cnt; j += T) {
            const K key = sk[j];
            int d = int((key >> shift) & 255);
            unsigned long long g = base[d] + (unsigned)(j - dstart[d]);
            kout[g] = key;
            vout[g] = sv[j];
        }
        __syncthreads();
        for (int d = tid; d < 256; d += T) base[d] += tcount[d];
        __syncthreads();
    }
}

template <class K, class V>
static constexpr size_t rs_down_smem() {
    constexpr int T = RsCfg<K, V>::threads, TILE = RsCfg<K, V>::tile;
    return 2 * size_t(TILE) * (sizeof(K) + sizeof(V)) + size_t(T / 32 + 2) * 256 * 4 + 32 * 4 + 256 * 8;
}
cudaError_t pack_text(const uint8_t* reads, size_t n, idx_t L, int dir, uint64_t* pk, cudaStream_t st) {
    const size_t nwords = n / 32 + 4;
    { k_pack_text<<<grid_for(nwords, 256), 256, 0, st>>>(reads, n, make_divl(uint32_t(L)), dir, nwords, pk); note_launch(); }
    return cudaGetLastError();
}

size_t radix_tmp_bytes(size_t n) {
    (void)n;
    return (size_t(256) * RS_MAX_CTAS + 9 * 256 + 64) * sizeof(unsigned long long);
}

template <class K, class V>
int radix_sort_pairs(K** k0, V** v0, K** k1, V** v1, size_t n, int lo_bit, int hi_bit, void* tmp,
                     size_t tmp_bytes, cudaStream_t st, bool skip_trivial) {
    constexpr int D = int(sizeof(K));
    if (hi_bit > 8 * D) hi_bit = 8 * D;
    if (n <= 1) return 0;
    if (tmp_bytes < radix_tmp_bytes(n)) return int(cudaErrorInvalidValue);
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(tmp);
    unsigned long long* gh = cnt + size_t(256) * RS_MAX_CTAS;
    unsigned long long* total = gh + 8 * 256;
    std::vector<unsigned long long> h(size_t(D) * 256, 0);
    if (skip_trivial) {
        cudaMemsetAsync(gh, 0, 8 * 256 * sizeof(unsigned long long), st);
        { k_digit_hist<K><<<grid_for(n, 256, 4), 256, 0, st>>>(*k0, n, gh); note_launch(); }
        cudaMemcpyAsync(h.data(), gh, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return int(e);
    }
    size_t tiles = (n + RS_TILE_MAX - 1) / RS_TILE_MAX;
    // one wave of resident CTAs: as many per SM as the downsweep's shared memory and registers
    // allow (a grid sized for more ran a second, partial wave on a fraction of the SMs)
    constexpr size_t smem = rs_down_smem<K, V>();
    const cudaError_t allowed = allow_smem<smem>(k_rs_downsweep<K, V>);
    if (allowed != cudaSuccess) return int(allowed);
    int dev = 0, sms = 152, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rs_downsweep<K, V>, RsCfg<K, V>::threads, smem) !=
            cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    size_t ctas = std::min<size_t>(tiles, std::min<size_t>(RS_MAX_CTAS, size_t(sms) * size_t(per_sm)));
    size_t part = ((tiles + ctas - 1) / ctas) * RS_TILE_MAX;
    ctas = (n + part - 1) / part;
    for (int d = lo_bit / 8; d * 8 < hi_bit; ++d) {
        bool trivial = false;
        for (int b = 0; b < 256; ++b)
            if (h[size_t(d) * 256 + b] == n) trivial = true;
        if (trivial) continue;
        { k_rs_upsweep<K><<<unsigned(ctas), RS_THREADS, 0, st>>>(*k0, n, 8 * d, part, cnt); note_launch(); }
        { k_rs_scan<<<256, RS_THREADS, 0, st>>>(cnt, unsigned(ctas), total); note_launch(); }
        // whole tiles are prefetched by 16-byte copies when both inputs are 16-byte aligned
        const int staged = (reinterpret_cast<uintptr_t>(*k0) % 16 == 0 && reinterpret_cast<uintptr_t>(*v0) % 16 == 0);
        { k_rs_downsweep<K, V><<<unsigned(ctas), RsCfg<K, V>::threads, smem, st>>>(*k0, *v0, *k1, *v1, n, 8 * d, part,
                                                                                   cnt, total, staged); note_launch(); }
        std::swap(*k0, *k1);
        std::swap(*v0, *v1);
    }
    return int(cudaGetLastError());
}

template int radix_sort_pairs<uint64_t, idx_t>(uint64_t**, idx_t**, uint64_t**, idx_t**, size_t, int, int, void*, size_t,
                                               cudaStream_t, bool);
template int radix_sort_pairs<uint32_t, idx_t>(uint32_t**, idx_t**, uint32_t**, idx_t**, size_t, int, int, void*, size_t,
                                               cudaStream_t, bool);

// ------------------------------------------------------------------------------ group ranks

constexpr int HT_THREADS = 256;
constexpr int HT_IPT = 8;
constexpr int HT_TILE = HT_THREADS * HT_IPT;

// per tile: max over i of (key[i] != key[i-1] ? i : 0), and the number of group starts
__global__ void k_head_tiles(const uint64_t* __restrict__ key, size_t n, unsigned long long* __restrict__ tmax,
                             unsigned long long* __restrict__ tcnt) {
    __shared__ unsigned long long smax[HT_THREADS / 32], scnt[HT_THREADS / 32];
    const size_t t0 = size_t(blockIdx.x) * HT_TILE;
    unsigned long long m = 0, c = 0;
    for (int j = threadIdx.x; j < HT_TILE; j += HT_THREADS) {
        size_t i = t0 + j;
        if (i >= n) break;
        bool f = (i == 0) || key[i] != key[i - 1];
        if (f) { m = i; c++; }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_down_sync(0xffffffffu, m, o));
        c += __shfl_down_sync(0xffffffffu, c, o);
    }
    if ((threadIdx.x & 31) == 0) { smax[threadIdx.x >> 5] = m; scnt[threadIdx.x >> 5] = c; }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long M = 0, Cn = 0;
        for (int w = 0; w < HT_THREADS / 32; ++w) { M = max(M, smax[w]); Cn += scnt[w]; }
        tmax[blockIdx.x] = M;
        tcnt[blockIdx.x] = Cn;
    }
}

// single CTA: exclusive max-scan of tile maxima (in place), total of tile counts into *groups
__global__ void k_head_carry(unsigned long long* __restrict__ tmax, const unsigned long long* __restrict__ tcnt,
                             size_t m, unsigned long long* __restrict__ groups) {
    __shared__ unsigned long long wv[32], carry, total;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) { carry = 0; total = 0; }
    __syncthreads();
    for (size_t base = 0; base < m; base += 1024) {
        size_t i = base + threadIdx.x;
        unsigned long long v = i < m ? tmax[i] : 0, x = v;
        unsigned long long c = i < m ? tcnt[i] : 0;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x = max(x, y);
        }
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
        if (lane == 31) wv[wid] = x;
        if (lane == 0) atomicAdd(&total, c);
        __syncthreads();
        unsigned long long pre = carry;
        for (int w = 0; w < wid; ++w) pre = max(pre, wv[w]);
        unsigned long long up = __shfl_up_sync(0xffffffffu, x, 1);
        unsigned long long excl = lane ? max(pre, up) : pre;
        if (i < m) tmax[i] = excl;
        __syncthreads();
        if (threadIdx.x == 1023) carry = max(pre, x);
        __syncthreads();
    }
    if (threadIdx.x == 0) *groups = total;
}

// head[i] = last group start <= i; rank[val[i]] = head[i]; kout[i] = head[i] << 32
// (kout != key: neighbouring threads still read key[i0-1])
template <class V>
__global__ void k_head_apply(const uint64_t* __restrict__ key, uint64_t* __restrict__ kout, const V* __restrict__ val,
                             size_t n, const unsigned long long* __restrict__ carry, uint32_t* __restrict__ rank) {
    __shared__ unsigned long long wv[HT_THREADS / 32];
    const size_t t0 = size_t(blockIdx.x) * HT_TILE;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // thread owns HT_IPT consecutive items
    const size_t i0 = t0 + size_t(threadIdx.x) * HT_IPT;
    unsigned long long h[HT_IPT];
    uint64_t prevk = (i0 > 0 && i0 < n) ? key[i0 - 1] : 0;
    unsigned long long run = 0;
    #pragma unroll
    for (int j = 0; j < HT_IPT; ++j) {
        size_t i = i0 + j;
        uint64_t kk = i < n ? key[i] : 0;
        bool f = i < n && (i == 0 || kk != prevk);
        if (f) run = i;
        h[j] = run;
        prevk = kk;
    }
    unsigned long long x = run;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = max(x, y);
    }
    if (lane == 31) wv[wid] = x;
    __syncthreads();
    unsigned long long pre = carry[blockIdx.x];
    for (int w = 0; w < wid; ++w) pre = max(pre, wv[w]);
    unsigned long long up = __shfl_up_sync(0xffffffffu, x, 1);
    unsigned long long excl = lane ? max(pre, up) : pre;
    #pragma unroll
    for (int j = 0; j < HT_IPT; ++j) {
        size_t i = i0 + j;
        if (i < n) {
            unsigned long long hd = max(excl, h[j]);
            rank[val[i]] = uint32_t(hd);
            kout[i] = uint64_t(hd) << 32;
        }
    }
}

// key[i] |= rank of the suffix h bases further (+1), or 0 when that lies past the read end
template <class V>
__global__ void k_second_keys(uint64_t* __restrict__ key, const V* __restrict__ val, size_t n, idx_t L, size_t h,
                              const uint32_t* __restrict__ rank) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        size_t p = val[i];
        size_t off = p % L;
        uint64_t second = (off + h < size_t(L)) ? uint64_t(rank[p + h]) + 1 : 0;
        key[i] |= second;
    }
}

template <class V>
__global__ void k_copy_vals(const V* __restrict__ v, size_t n, idx_t* __restrict__ sa) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) sa[i] = idx_t(v[i]);
}
// ------------------------------------------------------------------------------ elements and plan
//
// An element, highest bits first: kbits of the suffix's text (after the first d1 bits, padded with
// A past its end), min(length, head) in 5 bits, the position, the BWT symbol in 3 bits (0 = `$`,
// else the preceding base).  Comparing two elements of one first-level bucket as integers compares
// the suffixes' first `head` bases, end-of-read lowest, then the positions.

constexpr int kLenBits = 5, kSymBits = 3;
constexpr int kLocalSmall = 2560;           // buckets finished by a CTA of 128 threads
constexpr int kLocalLarge = 8192;           // ... of 256 threads; larger ones are split further
constexpr int kSplitTile = 8192;            // elements per tile of the partition passes
constexpr int kSplitThreads = 512;
constexpr int kMaxDigit = 11;               // bits of one partition pass
constexpr int kMaxWords = 9;                // 64-bit words of a suffix the networks compare
#ifdef PQ_IDX64
using kmer_int = unsigned long long;
#else
using kmer_int = unsigned;
#endif
constexpr int kMoreBits = 10;               // bits of one further split

struct MsdPlan {
    size_t n;
    DivL dl;
    int P;                  // position bits
    int d1, d2;             // bits of the two partition passes (d2 = 0: one pass)
    int kbits, head;        // text bits of an element's key; bases it and the first pass tell apart
    int S;                  // suffixes of at most S bases are sorted apart (0: none)
    int len_shift, key_shift;
};

// d1 and d2 by the bucket size aimed at: 600 to 1200 suffixes where there are enough of them to fill
// the chip (smaller: more counters and barriers per suffix; larger: buckets beyond the small
// kernel's 2560 under a skewed base composition), 400 at most for inputs of under 4 M suffixes,
// whose few buckets would otherwise leave most SMs idle.  One pass covers 2^11 buckets (its counters, and 4 elements
// a bucket and tile, the least that fills a sector).  In chunks the first pass takes all its 11 bits: a
// chunk is a run of its buckets.
static MsdPlan make_plan(size_t n, size_t nr, idx_t L, bool shorts, bool chunked) {
    MsdPlan p{};
    p.n = n;
    p.dl = make_divl(uint32_t(L));
    p.P = 1;
    while ((size_t(1) << p.P) < n) ++p.P;
    const size_t target = n < (size_t(1) << 22) ? 400 : 1200;
    int bt = 2;
    while (bt < 2 * kMaxDigit && (n >> bt) > target) ++bt;
    if (n < (size_t(1) << 22)) bt = std::min(bt, kMaxDigit);
    p.d1 = bt <= kMaxDigit ? bt : (chunked ? kMaxDigit : (bt + 1) / 2);
    p.d2 = bt - p.d1;
    p.kbits = std::min(64 - kLenBits - kSymBits - p.P, 62 - p.d1);
    if ((p.d1 + p.kbits) & 1) --p.kbits;
    p.head = (p.d1 + p.kbits) / 2;
    p.len_shift = kSymBits + p.P;
    p.key_shift = p.len_shift + kLenBits;
    // a string of m bases has about nr / 4^m equal suffixes of that length: those of more than 512
    // (half the suffixes at most, which bounds the memory they take: with a quarter 24 M suffixes of 12-base reads
    // took 1.55 ms, now 1.16; a quarter of shorter reads', which come to the static sort's fixed memory only)
    if (shorts)
        while (p.S < 7 && (L > 10 ? 2 : 4) * (p.S + 1) <= int(L) && 2 * p.S + 2 <= bt && (nr >> (2 * p.S + 2)) > 512) ++p.S;
    return p;
}

// words of the networks: bases from the partition's own on, 29 in the first word, 32 in the others
static int plan_words(const MsdPlan& p) {
    const int rest = int(p.dl.L) - (p.d1 + p.d2) / 2 - 29;
    return 1 + (rest > 0 ? (rest + 31) / 32 : 0);
}

// bases from text position p to the end of its read; positions of a 32-bit index take one 32-bit
// multiply-high by floor(2^32 / L): the quotient is short by at most one below 2^32
__device__ __forceinline__ int suffix_bases(size_t p, const DivL& dl) {
#ifdef PQ_IDX64
    return dl.L == 1 ? 1 : int(dl.L - uint32_t(p - div_l(p, dl) * dl.L));      // div_l: L of 2 and more
#else
    const uint32_t x = uint32_t(p), q = __umulhi(x, dl.m32), r = x - q * dl.L;
    return int((r >= dl.L ? 2 * dl.L : dl.L) - r);
#endif
}

// the element of the suffix at p (m bases, whose text starts the window x, preceded by the base
// `prev`) and its first-level digit
__device__ __forceinline__ uint64_t make_element(const MsdPlan& a, size_t p, int m, uint64_t x, int prev, bool dollar,
                                                 unsigned& digit) {
    const uint64_t xm = m < 32 ? x & (~uint64_t(0) << (64 - 2 * m)) : x;
    digit = unsigned(xm >> (64 - a.d1));
    const uint64_t key = (xm << a.d1) >> (64 - a.kbits);
    const int w = m < a.head ? m : a.head;
    return (key << a.key_shift) | (uint64_t(w) << a.len_shift) | (uint64_t(p) << kSymBits) |
           uint64_t(dollar ? 0 : prev + 1);
}

// A thread's 16 consecutive text positions from two words of the packed text: f(position, window,
// bases to the end of the read, preceding base, first of its read)
template <class F>
__device__ __forceinline__ void for_positions(const uint64_t* __restrict__ pk, size_t p0, size_t n, const DivL& dl, F f) {
    if (p0 >= n) return;
    const size_t w = p0 >> 5;
    const uint64_t a = pk[w], b = pk[w + 1];
    const int s0 = int(p0 & 31);                // 0 or 16
    int prev = s0 ? int(a >> (64 - 2 * s0)) & 3 : (w ? int(pk[w - 1]) & 3 : 0);
    int m = suffix_bases(p0, dl);
    #pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int sh = 2 * (s0 + j);
        const uint64_t x = sh ? ((a << sh) | (b >> (64 - sh))) : a;
        if (p0 + size_t(j) < n) f(j, p0 + size_t(j), x, m, prev, m == int(dl.L));
        prev = int(x >> 62);
        m = m == 1 ? int(dl.L) : m - 1;
    }
}

// exclusive scan of cnt[0, bins) into start[0, bins) by the whole CTA of T threads (bins a power of
// two; the caller synchronises before reading start); returns the total to every thread
template <int T>
__device__ __forceinline__ unsigned bins_exclusive(const unsigned* cnt, unsigned* start, int bins, unsigned* wsum) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = bins > T ? bins / T : 1;
    const int b0 = tid * per;
    unsigned mine = 0;
    if (b0 < bins)
        for (int i = 0; i < per; ++i) mine += cnt[b0 + i];
    unsigned x = mine;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned pre = 0, all = 0;
    #pragma unroll
    for (int w = 0; w < T / 32; ++w) {
        pre += w < warp ? wsum[w] : 0u;
        all += wsum[w];
    }
    unsigned run = pre + x - mine;
    if (b0 < bins)
        for (int i = 0; i < per; ++i) {
            const unsigned c = cnt[b0 + i];
            start[b0 + i] = run;
            run += c;
        }
    return all;
}

// ------------------------------------------------------------------------------ partition passes

// how many suffixes start with each d1-bit prefix (padded with A).  Bound by integer instructions: 16
// positions a thread from two 32-bit halves of the packed text; with 64-bit windows 113 M positions
// took 0.15 ms, now 0.08.
__global__ void __launch_bounds__(kSplitThreads) k_msd_hist(const uint64_t* __restrict__ pk, MsdPlan a,
                                                            unsigned long long* __restrict__ cnt) {
    __shared__ unsigned h[1 << kMaxDigit];
    const int bins = 1 << a.d1;
    for (int i = threadIdx.x; i < bins; i += kSplitThreads) h[i] = 0;
    __syncthreads();
    const size_t stride = size_t(gridDim.x) * kSplitThreads * 16;
    const uint32_t* const half = reinterpret_cast<const uint32_t*>(pk);     // the words' halves, lower first
    for (size_t p0 = (size_t(blockIdx.x) * kSplitThreads + threadIdx.x) * 16; p0 < a.n; p0 += stride) {
        const uint32_t w0 = half[(p0 >> 4) ^ 1], w1 = half[((p0 >> 4) + 1) ^ 1];
        const int left = int(a.n - p0 < 16 ? a.n - p0 : 16);
        int m = suffix_bases(p0, a.dl);
        #pragma unroll
        for (int j = 0; j < 16; ++j) {
            uint32_t past;
            asm("shr.u32 %0, %1, %2;" : "=r"(past) : "r"(0xffffffffu), "r"(2u * unsigned(m)));      // 0 from 32 on
            const uint32_t x = __funnelshift_l(w1, w0, 2 * j) & ~past;
            if (j < left) atomicAdd(&h[x >> (32 - a.d1)], 1u);
            m = m == 1 ? int(a.dl.L) : m - 1;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < bins; i += kSplitThreads)
        if (h[i]) atomicAdd(&cnt[i], (unsigned long long)h[i]);
}

// A chunk's bucket numbers: the first 6 bases (padded with A) above min(length, 6), in suffix order
constexpr int kBucketBases = 6;
constexpr int kBuckets = (1 << (2 * kBucketBases)) * 8;
__device__ __forceinline__ uint32_t bucket6(uint64_t x, int m) {
    const int w = m < kBucketBases ? m : kBucketBases;
    const uint32_t pre = uint32_t(x >> (64 - 2 * kBucketBases)) & (~0u << (2 * (kBucketBases - w)));
    return (pre << 3) | uint32_t(w);
}

// First pass: every suffix of more than S bases (of a chunk: whose 6-base bucket lies in
// [c0, c1)) as an element into its d1-bit bucket.  Bound by the 8 bytes written per suffix (the
// text is a quarter byte): a tile of 8192 positions is ranked with one shared-memory atomic a
// suffix, takes its place in every bucket with one global atomic a bucket, and leaves through
// shared memory in runs.  That, not the 8 bytes, takes the time: the ranking, the way through shared
// memory and their barriers; 113 M suffixes take 0.58 ms (0.65 with 64-bit windows), 0.16 at the rate of
// a copy.
struct MsdSmem {            // dynamic shared memory of the partition passes
    static constexpr size_t bins = size_t(1) << kMaxDigit;
    static constexpr size_t elems = size_t(kSplitTile) * 8;
    static constexpr size_t bytes(int bits, bool digits) {
        return elems + (size_t(1) << bits) * (sizeof(idx_t) + 4 + 4) + (digits ? size_t(kSplitTile) * 2 : 0);
    }
};

// With 32-bit Out only the positions are written (k_msd_gather makes elements of them later).
template <class Out>
__global__ void __launch_bounds__(kSplitThreads, 2) k_msd_text(const uint64_t* __restrict__ pk, MsdPlan a,
                                                               unsigned long long* __restrict__ cursor,
                                                               Out* __restrict__ out, uint32_t c0, uint32_t c1) {
    extern __shared__ __align__(16) unsigned char msd_smem[];
    __shared__ unsigned wsum[kSplitThreads / 32];
    const int bins = 1 << a.d1, tid = threadIdx.x;
    uint64_t* se = reinterpret_cast<uint64_t*>(msd_smem);
    idx_t* gb = reinterpret_cast<idx_t*>(se + kSplitTile);          // element j of bucket d to out[gb[d] + j]
    unsigned* cnt = reinterpret_cast<unsigned*>(gb + bins);
    unsigned* start = cnt + bins;
    uint16_t* sd = reinterpret_cast<uint16_t*>(start + bins);
    const uint32_t* const half = reinterpret_cast<const uint32_t*>(pk);     // the words' halves, lower first
    const bool chunk = c1 < uint32_t(kBuckets) || c0 > 0;
    const size_t tiles = (a.n + kSplitTile - 1) / kSplitTile;
    for (size_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        for (int i = tid; i < bins; i += kSplitThreads) cnt[i] = 0;
        __syncthreads();
        uint64_t v[16];
        unsigned dr[16];                        // digit << 16 | rank within the tile's bucket
        #pragma unroll
        for (int j = 0; j < 16; ++j) dr[j] = ~0u;
        const size_t p0 = t * kSplitTile + size_t(tid) * 16;
        if (p0 < a.n) {
            // three halves of the packed text hold the windows of the 16 positions
            const size_t w = p0 >> 4;
            const uint32_t w0 = half[w ^ 1], w1 = half[(w + 1) ^ 1], w2 = half[(w + 2) ^ 1];
            uint32_t prev = w ? half[(w - 1) ^ 1] & 3u : 0u;
            const int left = int(a.n - p0 < 16 ? a.n - p0 : 16);
            int m = suffix_bases(p0, a.dl);
            #pragma unroll
            for (int j = 0; j < 16; ++j) {
                uint32_t past0, past1;          // bits past the suffix's end
                asm("shr.u32 %0, %1, %2;" : "=r"(past0) : "r"(0xffffffffu), "r"(2u * unsigned(m)));        // 0 from 32 on
                asm("shr.u32 %0, %1, %2;" : "=r"(past1) : "r"(0xffffffffu), "r"(unsigned(max(2 * m - 32, 0))));
                const uint32_t x0 = __funnelshift_l(w1, w0, 2 * j), x1 = __funnelshift_l(w2, w1, 2 * j);
                const uint32_t y0 = x0 & ~past0, y1 = x1 & ~past1;
                bool in = j < left && m > a.S;
                if (chunk) {
                    const uint32_t c = bucket6(uint64_t(y0) << 32, m);
                    in = in && c >= c0 && c < c1;
                }
                if (in) {
                    const unsigned d = y0 >> (32 - a.d1);
                    const uint32_t k0 = __funnelshift_l(y1, y0, a.d1), k1 = y1 << a.d1;
                    const uint64_t key = (((uint64_t(k0) << 32) | k1) >> (64 - a.kbits)) << a.key_shift;
                    const uint32_t sym = m == int(a.dl.L) ? 0u : prev + 1u;
                    v[j] = key | (uint64_t(unsigned(min(m, a.head))) << a.len_shift) | (uint64_t(p0) << kSymBits) |
                           uint64_t((unsigned(j) << kSymBits) | sym);
                    dr[j] = (d << 16) | atomicAdd(&cnt[d], 1u);
                }
                prev = x0 >> 30;
                m = m == 1 ? int(a.dl.L) : m - 1;
            }
        }
        __syncthreads();
        const unsigned total = bins_exclusive<kSplitThreads>(cnt, start, bins, wsum);
        __syncthreads();
        for (int d = tid; d < bins; d += kSplitThreads) {
            const unsigned c = cnt[d];
            if (c) gb[d] = idx_t(atomicAdd(&cursor[d], (unsigned long long)c) - start[d]);
        }
        #pragma unroll
        for (int j = 0; j < 16; ++j)
            if (dr[j] != ~0u) {
                const unsigned q = start[dr[j] >> 16] + (dr[j] & 0xffffu);
                se[q] = v[j];
                sd[q] = uint16_t(dr[j] >> 16);
            }
        __syncthreads();
        #pragma unroll 4
        for (unsigned j = tid; j < total; j += kSplitThreads)
            out[idx_t(gb[sd[j]] + j)] = Out(sizeof(Out) == 8 ? se[j] : (se[j] >> kSymBits) & ((uint64_t(1) << a.P) - 1));
        __syncthreads();
    }
}

// Ranges [start, end) of elements to split by one digit each, in tiles of kSplitTile: tile0 is the
// exclusive scan of their tile counts (count + 1 entries).
struct MsdRanges {
    const unsigned long long* start;
    const unsigned long long* end;
    const unsigned* tile0;
    const int* shift;                   // a range's digit is (element >> (shift & 63)) & (2^bits - 1),
    int ushift;                         // with one shift for all when `shift` is null
    int count, bits;
    unsigned long long base;            // of starts and ends: element 0 of the array is theirs of `base`
};
__device__ __forceinline__ int range_of(const MsdRanges& r, unsigned tile) {
    int lo = 0, hi = r.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(r.tile0 + mid) <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(1024) k_msd_tiles(const unsigned long long* __restrict__ start,
                                                    const unsigned long long* __restrict__ end, int count,
                                                    unsigned* __restrict__ tile0) {
    __shared__ unsigned cnt[1 << kMaxDigit], ex[1 << kMaxDigit], wsum[32];
    for (int i = threadIdx.x; i < 1 << kMaxDigit; i += 1024)
        cnt[i] = i < count ? unsigned((end[i] - start[i] + kSplitTile - 1) / kSplitTile) : 0u;
    __syncthreads();
    const unsigned total = bins_exclusive<1024>(cnt, ex, 1 << kMaxDigit, wsum);
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += 1024) tile0[i] = ex[i];
    if (threadIdx.x == 0) tile0[count] = total;
}

// digit counts of every range, cnt[range << bits | digit]: a CTA takes consecutive tiles and adds
// its counts when the range changes
__global__ void __launch_bounds__(kSplitThreads) k_msd_count(const uint64_t* __restrict__ in, MsdRanges r,
                                                             unsigned long long* __restrict__ cnt) {
    __shared__ unsigned h[1 << kMaxDigit];
    const int bins = 1 << r.bits, tid = threadIdx.x;
    const unsigned tiles = r.tile0[r.count];
    const unsigned per = (tiles + gridDim.x - 1) / gridDim.x;
    const unsigned t0 = min(tiles, blockIdx.x * per), t1 = min(tiles, t0 + per);
    if (t0 >= t1) return;
    for (int i = tid; i < bins; i += kSplitThreads) h[i] = 0;
    __syncthreads();
    int q = range_of(r, t0);
    for (unsigned t = t0; t < t1; ++t) {
        if (t >= __ldg(r.tile0 + q + 1)) {
            __syncthreads();
            for (int i = tid; i < bins; i += kSplitThreads)
                if (h[i]) {
                    atomicAdd(&cnt[(size_t(q) << r.bits) + i], (unsigned long long)h[i]);
                    h[i] = 0;
                }
            q = range_of(r, t);
            __syncthreads();
        }
        const int shift = r.shift ? r.shift[q] & 63 : r.ushift;
        const size_t b = r.start[q] - r.base + size_t(t - r.tile0[q]) * kSplitTile;
        const size_t e = zmin(r.end[q] - r.base, b + kSplitTile);
        #pragma unroll 4
        for (size_t i = b + tid; i < e; i += kSplitThreads) atomicAdd(&h[(in[i] >> shift) & (bins - 1)], 1u);
    }
    __syncthreads();
    for (int i = tid; i < bins; i += kSplitThreads)
        if (h[i]) atomicAdd(&cnt[(size_t(q) << r.bits) + i], (unsigned long long)h[i]);
}

// The elements of the ranges' suffixes from their positions (element of `pos[i]` to out[i - base]).  Bound
// by the text's random sectors, one or two each.
__global__ void __launch_bounds__(kSplitThreads) k_msd_gather(const uint64_t* __restrict__ pk, MsdPlan a, const idx_t* __restrict__ pos,
                                                              MsdRanges r, uint64_t* __restrict__ out) {
    const unsigned tiles = r.tile0[r.count];
    for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int q = range_of(r, t);
        const size_t b = r.start[q] + size_t(t - __ldg(r.tile0 + q)) * kSplitTile, e = zmin(r.end[q], b + kSplitTile);
        #pragma unroll 4
        for (size_t i = b + threadIdx.x; i < e; i += kSplitThreads) {
            const size_t p = size_t(pos[i]);
            const int left = suffix_bases(p, a.dl);
            const int prev = p ? int(pk[(p - 1) >> 5] >> (62 - 2 * int((p - 1) & 31))) & 3 : 0;
            unsigned digit;
            out[i - size_t(r.base)] = make_element(a, p, left, window(pk, p), prev, left == int(a.dl.L), digit);
        }
    }
}

// Second pass: the elements of every range into its children (cursor[range << bits | digit] is
// their next place in `out`), a tile at a time as in the first pass; 8 bytes read and written per
// suffix.
__global__ void __launch_bounds__(kSplitThreads, 2) k_msd_split(const uint64_t* __restrict__ in, MsdRanges r,
                                                                unsigned long long* __restrict__ cursor,
                                                                uint64_t* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char msd_smem[];
    __shared__ unsigned wsum[kSplitThreads / 32];
    const int bins = 1 << r.bits, tid = threadIdx.x;
    uint64_t* se = reinterpret_cast<uint64_t*>(msd_smem);
    idx_t* gb = reinterpret_cast<idx_t*>(se + kSplitTile);          // element j of bucket d to out[gb[d] + j]
    unsigned* cnt = reinterpret_cast<unsigned*>(gb + bins);
    unsigned* start = cnt + bins;
    const unsigned tiles = r.tile0[r.count];
    constexpr int kPer = kSplitTile / kSplitThreads;
    for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int q = range_of(r, t);
        const int shift = r.shift ? r.shift[q] & 63 : r.ushift;
        const size_t b = r.start[q] - r.base + size_t(t - __ldg(r.tile0 + q)) * kSplitTile;
        const int m = int(zmin(size_t(kSplitTile), r.end[q] - r.base - b));
        uint64_t v[kPer];
        #pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int i = tid + j * kSplitThreads;
            v[j] = i < m ? in[b + i] : 0;
        }
        for (int i = tid; i < bins; i += kSplitThreads) cnt[i] = 0;
        __syncthreads();
        unsigned rk[kPer];
        #pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (tid + j * kSplitThreads < m) rk[j] = atomicAdd(&cnt[unsigned(v[j] >> shift) & (bins - 1)], 1u);
        __syncthreads();
        bins_exclusive<kSplitThreads>(cnt, start, bins, wsum);
        __syncthreads();
        for (int d = tid; d < bins; d += kSplitThreads) {
            const unsigned c = cnt[d];
            if (c) gb[d] = idx_t(atomicAdd(&cursor[(size_t(q) << r.bits) + d], (unsigned long long)c) - start[d]);
        }
        #pragma unroll
        for (int j = 0; j < kPer; ++j)
            if (tid + j * kSplitThreads < m) se[start[unsigned(v[j] >> shift) & (bins - 1)] + rk[j]] = v[j];
        __syncthreads();
        #pragma unroll 4
        for (int j = tid; j < m; j += kSplitThreads) {
            const uint64_t e = se[j];
            out[idx_t(gb[unsigned(e >> shift) & (bins - 1)] + idx_t(j))] = e;
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------ buckets

// A bucket to finish: elements [start, start + size), whose suffixes share their first `off` bases;
// id (off = 0 only) is its d1 + d2-bit prefix.
struct __align__(16) MsdBucket {
    unsigned long long start;
    unsigned size;
    unsigned id_off;                    // off << 22 | id
};
constexpr int kIdBits = 22;

// Device counters of one sort
struct MsdCounters {
    unsigned long long small, large, more, mid, big, huge;      // list lengths (see MsdLists)
    unsigned long long next_small, next_large;                  // next bucket to take
};
// small, large: buckets for the two local kernels; more: buckets larger than both; mid, big, huge:
// groups of 33..128, 129..1024 and more suffixes equal in all bases of their elements
struct MsdLists {
    MsdBucket *small, *large, *more;
    unsigned long long *mid, *big, *huge;       // start << 24 | bases known equal << 14 | size
    unsigned long long cap_more, cap_mid, cap_big, cap_huge;
    MsdCounters* c;
};

__device__ __forceinline__ void list_bucket(const MsdLists& G, int cls, const MsdBucket& b) {
    const int lane = threadIdx.x & 31;
    #pragma unroll
    for (int z = 0; z < 3; ++z) {
        const unsigned peers = __ballot_sync(0xffffffffu, cls == z);
        if (!peers) continue;
        unsigned long long* c = z == 0 ? &G.c->small : (z == 1 ? &G.c->large : &G.c->more);
        MsdBucket* l = z == 0 ? G.small : (z == 1 ? G.large : G.more);
        unsigned long long at = 0;
        if (lane == __ffs(peers) - 1) at = atomicAdd(c, (unsigned long long)__popc(peers));
        at = __shfl_sync(0xffffffffu, at, __ffs(peers) - 1) + __popc(peers & ((1u << lane) - 1u));
        if (cls == z && (z != 2 || at < G.cap_more)) l[at] = b;
    }
}

// The children of first-level bucket first + blockIdx.x: from their counts (of long suffixes, or with
// `incl` of all) and the short suffixes of each (which come first in it), the place of each child's
// long suffixes: lstart, kept, and, from `row0` on, cursor, which the next pass advances; with `lists`,
// the non-empty ones listed by size.
constexpr int kScanThreads = 256;
__global__ void __launch_bounds__(kScanThreads) k_msd_children(const unsigned long long* __restrict__ cnt,
                                                               const unsigned long long* __restrict__ shorts, int bits,
                                                               int incl, const unsigned long long* __restrict__ base,
                                                               unsigned long long* __restrict__ lstart,
                                                               unsigned long long* __restrict__ cursor, int lists,
                                                               MsdLists G, unsigned first = 0, unsigned long long row0 = 0) {
    __shared__ unsigned long long wsum[kScanThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int bins = 1 << bits;
    const size_t c0 = size_t(first + blockIdx.x) << bits;
    const int per = bins > kScanThreads ? bins / kScanThreads : 1;
    const int b0 = tid * per;
    unsigned long long mine = 0;
    for (int i = 0; i < per; ++i)
        if (b0 + i < bins) mine += cnt[c0 + b0 + i] + (shorts && !incl ? shorts[c0 + b0 + i] : 0ull);
    unsigned long long x = mine;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned long long run = x - mine + (base ? base[first + blockIdx.x] : 0ull);
    for (int w = 0; w < warp; ++w) run += wsum[w];
    for (int i = 0; i < per; ++i) {
        int cls = -1;
        MsdBucket b{};
        if (b0 + i < bins) {
            const size_t c = c0 + b0 + i;
            const unsigned long long sh = shorts ? shorts[c] : 0ull;
            const unsigned long long all = cnt[c] + (incl ? 0ull : sh), longs = all - sh;
            lstart[c] = run + sh;
            cursor[c] = run + sh - row0;
            if (lists && longs) {
                cls = longs <= kLocalSmall ? 0 : (longs <= kLocalLarge ? 1 : 2);
                b.start = run + sh - row0;
                b.size = unsigned(longs < 0xffffffffull ? longs : 0xffffffffull);
                b.id_off = unsigned(c);
            }
            run += all;
        }
        if (lists) list_bucket(G, cls, b);
    }
}

// ------------------------------------------------------------------------------ short suffixes
//
// The suffixes of m <= S bases: every string has about nr / 4^m equal copies, in read order.  Sorted
// by a stable radix sort (from read order) on the string's preorder number in the trie of S bases,
// which is suffix order: for bases s_0 .. s_{m-1}, sum_i (1 + s_i T(S - 1 - i)) with T(h) the nodes
// of a subtree of height h, i.e. (4 v - sum s_i) / 3 + m with v the padded value.

constexpr int kShortSym = 20;           // a short suffix's BWT symbol, above the sorted key bits

__global__ void k_short_keys(const uint64_t* __restrict__ pk, size_t nr, idx_t L, int S, uint32_t* __restrict__ key,
                             idx_t* __restrict__ val) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nr * size_t(S); i += stride) {
        const size_t r = i / unsigned(S);
        const int m = int(i - r * unsigned(S)) + 1;
        const size_t p = r * size_t(L) + size_t(L) - size_t(m);
        const uint32_t v = uint32_t((window(pk, p) & (~uint64_t(0) << (64 - 2 * m))) >> (64 - 2 * S));
        const uint32_t sum = uint32_t(__popc(v & 0x55555555u)) + 2u * uint32_t(__popc(v & 0xaaaaaaaau));
        const uint32_t code = (4u * v - sum) / 3u + uint32_t(m);
        const uint32_t sym = m == int(L) ? 0u : (uint32_t(pk[(p - 1) >> 5] >> (62 - 2 * int((p - 1) & 31))) & 3u) + 1u;
        key[i] = code | (sym << kShortSym);
        val[i] = idx_t(p);
    }
}

// the bucket of a short suffix at p (its bases, padded with A)
__device__ __forceinline__ size_t short_bucket(const uint64_t* __restrict__ pk, size_t p, const DivL& dl, int bits) {
    const int m = suffix_bases(p, dl);
    return size_t((window(pk, p) & (~uint64_t(0) << (64 - 2 * m))) >> (64 - bits));
}

// per bucket: how many short suffixes it has and the index of the first of them (they are
// consecutive); every run of equal strings adds its ends
__global__ void k_short_runs(const uint64_t* __restrict__ pk, const uint32_t* __restrict__ key,
                             const idx_t* __restrict__ val, size_t m, DivL dl, int bits,
                             unsigned long long* __restrict__ count, unsigned long long* __restrict__ first) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    constexpr uint32_t mask = (1u << kShortSym) - 1u;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += stride) {
        const uint32_t k = key[i] & mask;
        const bool head = i == 0 || (key[i - 1] & mask) != k, tail = i + 1 == m || (key[i + 1] & mask) != k;
        if (!head && !tail) continue;
        const size_t b = short_bucket(pk, size_t(val[i]), dl, bits);
        if (head) {
            atomicMin(&first[b], (unsigned long long)i);
            atomicAdd(&count[b], 0ull - (unsigned long long)i);
        }
        if (tail) atomicAdd(&count[b], (unsigned long long)i + 1ull);
    }
}

// the rows of the short suffixes: before their bucket's long ones; those of at least k bases also
// belong to a k-mer (k <= S only: kt null otherwise), and where it has them (kx_bits) its rows' next
// bases, padded with A as in an element
__global__ void k_short_place(const uint64_t* __restrict__ pk, const uint32_t* __restrict__ key,
                              const idx_t* __restrict__ val, size_t m, DivL dl, int bits,
                              const unsigned long long* __restrict__ count, const unsigned long long* __restrict__ first,
                              const unsigned long long* __restrict__ lstart, idx_t* __restrict__ sa,
                              uint8_t* __restrict__ bwt, idx_t* __restrict__ kt, int k, uint16_t* __restrict__ kx, int kx_bits) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += stride) {
        const idx_t p = val[i];
        const size_t b = short_bucket(pk, size_t(p), dl, bits);
        const size_t row = size_t(lstart[b] - count[b] + (i - first[b]));
        sa[row] = p;
        if (bwt) bwt[row] = uint8_t(key[i] >> kShortSym);
        const int left = suffix_bases(size_t(p), dl);
        if (kt && left >= k) {
            const uint64_t x = window(pk, size_t(p)) & (~uint64_t(0) << (64 - 2 * left));
            const size_t c = size_t(x >> (64 - 2 * k));
            if (kx_bits) kx[row] = uint16_t((x << (2 * k)) >> (64 - kx_bits));
            atomicMin(reinterpret_cast<kmer_int*>(kt + 2 * c), kmer_int(row));
            atomicMax(reinterpret_cast<kmer_int*>(kt + 2 * c + 1), kmer_int(row));
        }
    }
}

// ------------------------------------------------------------------------------ networks
//
// Suffixes are compared by W 64-bit words of their bases (zero past the end: padded with A), then
// by a tail that holds the length and what breaks ties.

// a < b on (w[0..W-1], tail) as one unsigned multi-word number: the borrow out of the
// subtraction a - b, least significant word first, in one chain of subtract-with-borrow
// instructions (no branches; the chain must sit in one asm statement to keep the carry flag).
template <int W, class Tail>
struct SortItem {
    uint64_t w[W];              // w[0] starts with the segment number
    Tail tail;
};
template <int W>
__device__ __forceinline__ bool item_less(const SortItem<W, uint32_t>& a, const SortItem<W, uint32_t>& b);
template <int W>
__device__ __forceinline__ bool item_less(const SortItem<W, uint64_t>& a, const SortItem<W, uint64_t>& b);

#define PQ_S1 "subc.cc.u64 t, %3, %4;\n\t"
#define PQ_S2 PQ_S1 "subc.cc.u64 t, %5, %6;\n\t"
#define PQ_S3 PQ_S2 "subc.cc.u64 t, %7, %8;\n\t"
#define PQ_S4 PQ_S3 "subc.cc.u64 t, %9, %10;\n\t"
#define PQ_S5 PQ_S4 "subc.cc.u64 t, %11, %12;\n\t"
#define PQ_S6 PQ_S5 "subc.cc.u64 t, %13, %14;\n\t"
#define PQ_S7 PQ_S6 "subc.cc.u64 t, %15, %16;\n\t"
#define PQ_S8 PQ_S7 "subc.cc.u64 t, %17, %18;\n\t"
#define PQ_S9 PQ_S8 "subc.cc.u64 t, %19, %20;\n\t"
#define PQ_WORD(j) "l"(a.w[j]), "l"(b.w[j])
#define PQ_A1 PQ_WORD(0)
#define PQ_A2 PQ_WORD(1), PQ_A1
#define PQ_A3 PQ_WORD(2), PQ_A2
#define PQ_A4 PQ_WORD(3), PQ_A3
#define PQ_A5 PQ_WORD(4), PQ_A4
#define PQ_A6 PQ_WORD(5), PQ_A5
#define PQ_A7 PQ_WORD(6), PQ_A6
#define PQ_A8 PQ_WORD(7), PQ_A7
#define PQ_A9 PQ_WORD(8), PQ_A8
#define PQ_LESS(W)                                                                                                  \
    template <>                                                                                                     \
    __device__ __forceinline__ bool item_less<W>(const SortItem<W, uint32_t>& a, const SortItem<W, uint32_t>& b) {  \
        unsigned r;                                                                                                 \
        asm("{\n\t.reg .u64 t;\n\t.reg .u32 s, z;\n\tmov.u32 z, 0;\n\tsub.cc.u32 s, %1, %2;\n\t" PQ_S##W            \
            "subc.u32 %0, z, z;\n\t}"                                                                               \
            : "=r"(r) : "r"(a.tail), "r"(b.tail), PQ_A##W);                                                         \
        return r != 0;                                                                                              \
    }                                                                                                               \
    template <>                                                                                                     \
    __device__ __forceinline__ bool item_less<W>(const SortItem<W, uint64_t>& a, const SortItem<W, uint64_t>& b) {  \
        unsigned r;                                                                                                 \
        asm("{\n\t.reg .u64 t;\n\t.reg .u32 z;\n\tmov.u32 z, 0;\n\tsub.cc.u64 t, %1, %2;\n\t" PQ_S##W               \
            "subc.u32 %0, z, z;\n\t}"                                                                               \
            : "=r"(r) : "l"(a.tail), "l"(b.tail), PQ_A##W);                                                         \
        return r != 0;                                                                                              \
    }
PQ_LESS(1)
PQ_LESS(2)
PQ_LESS(3)
PQ_LESS(4)
PQ_LESS(5)
PQ_LESS(6)
PQ_LESS(7)
PQ_LESS(8)
PQ_LESS(9)
#undef PQ_LESS
#undef PQ_WORD
#undef PQ_S1
#undef PQ_S2
#undef PQ_S3
#undef PQ_S4
#undef PQ_S5
#undef PQ_S6
#undef PQ_S7
#undef PQ_S8
#undef PQ_S9
#undef PQ_A1
#undef PQ_A2
#undef PQ_A3
#undef PQ_A4
#undef PQ_A5
#undef PQ_A6
#undef PQ_A7
#undef PQ_A8
#undef PQ_A9

// The bases of the suffix at p (m bases to its end) from base `from` on, 16 to a word, first base
// highest, zero past the end; mask[i] has the bits of word i that are bases of the suffix.  Only
// words of the text that hold such bases are loaded.
template <int W>
__device__ __forceinline__ void suffix_text(const uint64_t* __restrict__ pk, size_t p, int m, int from, uint32_t (&x)[2 * W],
                                            uint32_t (&mask)[2 * W]) {
    const int rem = max(m - from, 0);
    const size_t q = p + size_t(from);
    const uint64_t* t = pk + (q >> 5);
    const int s = int(q & 31), held = rem + s;              // bases from the first word's start
    uint32_t r[2 * W + 2];
    #pragma unroll
    for (int j = 0; j <= W; ++j) {
        uint64_t v = 0;
        if (rem > 0 && held > 32 * j) v = t[j];
        r[2 * j] = uint32_t(v >> 32);
        r[2 * j + 1] = uint32_t(v);
    }
    const bool odd = s >= 16;
    #pragma unroll
    for (int i = 0; i <= 2 * W; ++i) r[i] = odd ? r[i + 1] : r[i];
    #pragma unroll
    for (int i = 0; i < 2 * W; ++i) {
        const uint32_t v = uint32_t(max(2 * rem - 32 * i, 0));
        uint32_t past;
        asm("shr.u32 %0, %1, %2;" : "=r"(past) : "r"(0xffffffffu), "r"(v));     // 0 from 32 on
        mask[i] = ~past;
        x[i] = __funnelshift_l(r[i + 1], r[i], 2 * s) & mask[i];
    }
}

// The same as W 64-bit words behind a segment number of SEG bits: (64 - SEG) / 2 bases in the first,
// 32 in each other.
template <int W, int SEG>
__device__ __forceinline__ void pack_words(const uint32_t (&x)[2 * W], uint32_t seg, uint64_t (&w)[W]) {
    constexpr int kFirst = 2 * ((64 - SEG) / 2);            // text bits of the first word
    uint64_t y[W];
    #pragma unroll
    for (int j = 0; j < W; ++j) y[j] = (uint64_t(x[2 * j]) << 32) | x[2 * j + 1];
    if constexpr (SEG == 0) {
        #pragma unroll
        for (int j = 0; j < W; ++j) w[j] = y[j];
    } else {
        w[0] = (uint64_t(seg) << (64 - SEG)) | ((y[0] >> (64 - kFirst)) << (64 - SEG - kFirst));
        #pragma unroll
        for (int j = 1; j < W; ++j) w[j] = (y[j - 1] << kFirst) | (y[j] >> (64 - kFirst));
    }
}
template <int W, int SEG>
__device__ __forceinline__ void sort_words(const uint64_t* __restrict__ pk, size_t p, int m, int from, uint32_t seg,
                                           uint64_t (&w)[W]) {
    uint32_t x[2 * W], mask[2 * W];
    suffix_text<W>(pk, p, m, from, x, mask);
    pack_words<W, SEG>(x, seg, w);
}

// ascending bitonic sort of one item a lane; lanes from `len` on hold the largest items
__device__ __forceinline__ bool item_less(uint64_t a, uint64_t b) { return a < b; }
__device__ __forceinline__ uint64_t item_xor(uint64_t a, int j) { return __shfl_xor_sync(0xffffffffu, a, j); }
template <int W>
__device__ __forceinline__ SortItem<W, uint64_t> item_xor(const SortItem<W, uint64_t>& a, int j) {
    SortItem<W, uint64_t> o;
    #pragma unroll
    for (int q = 0; q < W; ++q) o.w[q] = __shfl_xor_sync(0xffffffffu, a.w[q], j);
    o.tail = __shfl_xor_sync(0xffffffffu, a.tail, j);
    return o;
}
template <class Item>
__device__ __forceinline__ void warp_sort(Item& it, int len, int lane) {
    #pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
        if (k > 2 && len <= (k >> 1)) break;
        #pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            const Item o = item_xor(it, j);
            const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
            if (keep_min == item_less(o, it)) it = o;
        }
    }
}

// ------------------------------------------------------------------------------ buckets in shared memory

struct MsdLocal {
    MsdPlan plan;
    const uint64_t* pk;
    uint64_t* buf;                      // the buckets' elements
    const MsdBucket* list;
    const unsigned long long* count;
    unsigned long long* next;
    MsdLists G;
    idx_t* sa;                          // rows of element 0 on
    uint8_t* bwt;                       // or null
    idx_t* kt;                          // k-mer table, or null
    uint16_t* kx;                       // every row's next bases, or null: kx_bits bits of an element
    int kx_bits, kx_shift;              // from bit kx_shift on
    int kmer_k;
    int kmer_spans;                     // a k-mer's rows may lie in several buckets
    size_t row0;                        // suffix-array row of element 0
    int more_bits;                      // text bits of a rebuilt element's key (off > 0)
};

constexpr int kLocalBits = 11, kLocalBins = 1 << kLocalBits;      // two 16-bit counters to a word

// exclusive scan of the packed counters, in place, by the CTA's T threads (the caller synchronises
// before reading them)
template <int T>
__device__ __forceinline__ void packed_exclusive(unsigned* cnt, unsigned* wsum) {
    constexpr int kPer = kLocalBins / 2 / T;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned v[kPer], mine = 0;
    #pragma unroll
    for (int i = 0; i < kPer; ++i) {
        v[i] = cnt[tid * kPer + i];
        mine += (v[i] & 0xffffu) + (v[i] >> 16);
    }
    unsigned x = mine;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned run = x - mine;
    #pragma unroll
    for (int w = 0; w < T / 32; ++w) run += w < warp ? wsum[w] : 0u;
    #pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const unsigned lo = v[i] & 0xffffu;
        cnt[tid * kPer + i] = run | ((run + lo) << 16);
        run += lo + (v[i] >> 16);
    }
}

// first set bit of the boundary mask above slot j (there is one at the bucket's end)
__device__ __forceinline__ int next_boundary(const unsigned* bm, int j) {
    int w = (j + 1) >> 5;
    unsigned x = bm[w] & (~0u << ((j + 1) & 31));
    while (!x) x = bm[++w];
    return 32 * w + __ffs(x) - 1;
}

// ascending sort of e[0, m) by the `threads` threads of a warp or a CTA (t: this one's number):
// the bitonic network whose comparators all point up (a mirrored first step per merge), so that
// positions past m act as the largest and are skipped
template <class Sync>
__device__ __forceinline__ void smem_sort(uint64_t* e, int m, int t, int threads, Sync sync) {
    auto exchange = [&](int a, int b) {
        if (b >= m) return;
        const uint64_t x = e[a], y = e[b];
        if (y < x) {
            e[a] = y;
            e[b] = x;
        }
    };
    for (int k = 2; k < 2 * m; k <<= 1) {
        const int half = k >> 1, pairs = (m + k - 1) / k * half;
        for (int i = t; i < pairs; i += threads) {
            const int q = i / half, o = i - q * half;
            exchange(q * k + o, q * k + k - 1 - o);
        }
        sync();
        for (int j = half >> 1; j > 0; j >>= 1) {
            for (int i = t; i < pairs; i += threads) {
                const int a = ((i & ~(j - 1)) << 1) | (i & (j - 1));
                exchange(a, a + j);
            }
            sync();
        }
    }
}

// One bucket per CTA and turn.  Bound by instruction issue (the networks) and the gather of each
// suffix's text, about two sectors.  The elements are split by their next 11 bits into
// sub-buckets (counted and placed with shared-memory atomics; a bit mask marks where each starts),
// then every warp walks a stretch of sub-buckets: as many consecutive whole ones as fit 32 lanes
// are sorted by one bitonic network on (sub-bucket, bases, length, position).  Sub-buckets of more
// than 32 are first sorted by their elements; suffixes equal in all bases of those, if still more
// than 32, are listed for the kernels of larger groups, in order of position.
//
// A sub-bucket mostly holds the suffixes of one genome locus, equal up to their ends but for a few
// sequencing errors.  So the network does not carry their bases: every suffix is compared with the
// longest of its sub-bucket, the positions where any in the warp differs from its longest (within
// its length) are collected with one OR over the warp per word, and only the bases there, in order,
// enter the key.  Two suffixes of a sub-bucket that differ within both lengths differ at one of
// those positions, and past the end of the shorter one its bases there read A, so (those bases,
// length, position) is their order.  One 64-bit key holds 8 or so such positions beside length and
// position, two hold 27; only beyond that does the network carry all W words.
//
// Measured, one direction of 123 M suffixes of 100-base reads (32-bit positions): the whole sort 4.9
// ms, 3.3 of them here, against 8.0 ms for four radix passes of 14-base keys, group lists and
// refinement networks of all words; of 1.13 G suffixes (64-bit): 50 ms, 33 here, against 95.
template <int W, int CAP, int T>
__global__ void __launch_bounds__(T, T == 128 ? (W <= 4 ? 8 : 6) : 3) k_msd_local(MsdLocal a) {
    extern __shared__ __align__(16) unsigned char msd_smem[];
    uint64_t* se = reinterpret_cast<uint64_t*>(msd_smem);
    unsigned* cnt = reinterpret_cast<unsigned*>(se + CAP);
    unsigned* bm = cnt + kLocalBins / 2;                    // [CAP / 32 + 2]
    constexpr int kOver = CAP / 33 + 1;
    __shared__ unsigned s_over[kOver], wsum[T / 32], s_diff[2], s_item;
    __shared__ int s_nover, s_nhuge;
    __shared__ unsigned s_huge[CAP / 1025 + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = T / 32;
    const MsdPlan& P = a.plan;
    const uint64_t pos_mask = (uint64_t(1) << P.P) - 1;
    const int len_bits = 32 - __clz(int(P.dl.L));
    const unsigned items = unsigned(*a.count);
    while (true) {
        if (tid == 0) {
            s_item = unsigned(atomicAdd(a.next, 1ull));
            s_diff[0] = s_diff[1] = 0;
            s_nover = s_nhuge = 0;
        }
        __syncthreads();
        const unsigned item = s_item;
        if (item >= items) break;
        const MsdBucket bk = a.list[item];
        const int m = int(bk.size), off = int(bk.id_off >> kIdBits);
        uint64_t* const in = a.buf + bk.start;
        for (int i = tid; i < kLocalBins / 2; i += T) cnt[i] = 0;
        const int full = off ? a.more_bits / 2 : P.head;        // length field of a suffix that goes on
        // the lowest bit of the split, and the bases every sub-bucket then shares
        int shift, from;
        if (CAP == kLocalSmall) {                   // the bits below the partition's own
            shift = max(P.key_shift + P.kbits - P.d2 - kLocalBits, P.key_shift);
            __syncthreads();
        } else {                                    // the highest differing ones
            const uint64_t e0 = in[0];
            uint64_t diff = 0;
            for (int j = tid; j < m; j += T) diff |= in[j] ^ e0;
            const unsigned lo = __reduce_or_sync(0xffffffffu, unsigned(diff));
            const unsigned hi = __reduce_or_sync(0xffffffffu, unsigned(diff >> 32));
            if (lane == 0) {
                if (lo) atomicOr(&s_diff[0], lo);
                if (hi) atomicOr(&s_diff[1], hi);
            }
            __syncthreads();
            diff = (uint64_t(s_diff[1]) << 32) | s_diff[0];
            const int hb = diff ? 63 - __clzll((long long)diff) : -1;
            const bool goes_on = int((e0 >> P.len_shift) & 31u) == full;
            shift = hb - (kLocalBits - 1);
            if (hb >= P.key_shift) shift = max(shift, P.key_shift);
            else if (hb >= P.len_shift) shift = P.len_shift;
            else if (goes_on || hb < 0) shift = 63;             // equal heads: one sub-bucket
            else shift = max(shift, 0);                         // equal strings: by position
        }
        if (shift < P.key_shift || shift == 63) from = off + full;
        else if (off) from = off + min(a.more_bits, P.key_shift + P.kbits - shift) / 2;
        else from = (P.d1 + P.key_shift + P.kbits - shift) / 2;
        auto bin_of = [&](uint64_t e) { return unsigned(e >> shift) & unsigned(kLocalBins - 1); };
        for (int j = tid; j < m; j += T) {
            const unsigned q = bin_of(in[j]);
            atomicAdd(&cnt[q >> 1], q & 1u ? 0x10000u : 1u);
        }
        __syncthreads();
        packed_exclusive<T>(cnt, wsum);
        __syncthreads();
        for (int j = tid; j < m; j += T) {
            const uint64_t e = in[j];
            const unsigned q = bin_of(e), half = 16 * (q & 1u);
            se[(atomicAdd(&cnt[q >> 1], 1u << half) >> half) & 0xffffu] = e;
        }
        __syncthreads();
        const int words = m / 32 + 1;
        for (int w = warp; w < words; w += NW) {
            const int j = 32 * w + lane;
            bool b = j == m;
            if (j < m) b = j == 0 || bin_of(se[j]) != bin_of(se[j - 1]);
            const unsigned x = __ballot_sync(0xffffffffu, b);
            if (lane == 0) bm[w] = x;
        }
        if (tid == 0) bm[words] = 0;
        __syncthreads();
        // sub-buckets of more than 32: only the last one that starts in a mask word can be
        for (int w = tid; w < words; w += T) {
            const unsigned x = bm[w];
            if (!x) continue;
            const int j = 32 * w + 31 - __clz(x);
            if (j >= m) continue;
            const int g = next_boundary(bm, j) - j;
            if (g > 32) s_over[atomicAdd(&s_nover, 1)] = (unsigned(j) << 16) | unsigned(g);
        }
        __syncthreads();
        const int nover = s_nover;
        if (nover) {
            for (int i = warp; i < nover; i += NW) {
                const int j = int(s_over[i] >> 16), g = int(s_over[i] & 0xffffu);
                if (g <= 256) smem_sort(se + j, g, lane, 32, [] { __syncwarp(); });
            }
            __syncthreads();
            for (int i = 0; i < nover; ++i) {
                const int j = int(s_over[i] >> 16), g = int(s_over[i] & 0xffffu);
                if (g > 256) smem_sort(se + j, g, tid, T, [] { __syncthreads(); });
            }
            // their own sub-buckets: suffixes that go on past equal heads; ended ones are in order
            for (int i = warp; i < nover; i += NW) {
                const int j = int(s_over[i] >> 16), g = int(s_over[i] & 0xffffu);
                for (int q = lane; q < g; q += 32) {
                    const uint64_t e = se[j + q] >> P.len_shift;
                    if (q == 0 || e != (se[j + q - 1] >> P.len_shift) || int(e & 31u) < full)
                        atomicOr(&bm[(j + q) >> 5], 1u << ((j + q) & 31));
                }
            }
            __syncthreads();
            for (int w = tid; w < words; w += T) {
                const unsigned x = bm[w];
                if (!x) continue;
                const int j = 32 * w + 31 - __clz(x);
                if (j >= m) continue;
                const int g = next_boundary(bm, j) - j;
                if (g <= 32) continue;
                const int cls = g <= 128 ? 0 : (g <= 1024 ? 1 : 2);
                unsigned long long* c = cls == 0 ? &a.G.c->mid : (cls == 1 ? &a.G.c->big : &a.G.c->huge);
                unsigned long long* l = cls == 0 ? a.G.mid : (cls == 1 ? a.G.big : a.G.huge);
                const unsigned long long cap = cls == 0 ? a.G.cap_mid : (cls == 1 ? a.G.cap_big : a.G.cap_huge);
                const unsigned long long at = atomicAdd(c, 1ull);
                if (at < cap)
                    l[at] = ((bk.start + (unsigned long long)j) << 24) | ((unsigned long long)(off + full) << 14) |
                            (unsigned long long)g;
                if (cls == 2) s_huge[atomicAdd(&s_nhuge, 1)] = (unsigned(j) << 16) | unsigned(g);
            }
            __syncthreads();
            // groups that come back with new elements leave theirs in place
            for (int i = 0; i < s_nhuge; ++i) {
                const int j = int(s_huge[i] >> 16), g = int(s_huge[i] & 0xffffu);
                for (int q = tid; q < g; q += T) in[j + q] = se[j + q];
            }
        }
        // every warp's stretch of slots: the sub-buckets that start in it, 32 lanes at a time
        const int stretch = (m + NW - 1) / NW;
        const int r1 = min(m, (warp + 1) * stretch);
        int cur = warp * stretch;
        if (cur < r1 && !((bm[cur >> 5] >> (cur & 31)) & 1u)) cur = next_boundary(bm, cur);
        while (cur < r1) {
            // boundaries at slots cur + 1 .. cur + 32 as bits 0 .. 31
            const int w = (cur + 1) >> 5;
            unsigned x = __funnelshift_r(bm[w], bm[w + 1], (cur + 1) & 31);
            const int room = r1 - cur;                          // sub-buckets from slot r1 on are the next warp's
            if (room <= 32) {
                const unsigned low = (1u << (room - 1)) - 1u;
                const unsigned high = x & ~low;
                x = (x & low) | (high & (0u - high));
            }
            if (!x) {                                           // a listed group
                cur = next_boundary(bm, cur);
                continue;
            }
            const int len = 32 - __clz(x);
            const bool single = ((x >> lane) & 1u) && (lane == 0 || ((x >> (lane - 1)) & 1u));
            const bool need = lane < len && !single;
            if (__any_sync(0xffffffffu, need)) {
                const uint64_t e = lane < len ? se[cur + lane] : 0;
                const uint64_t p = (e >> kSymBits) & pos_mask;
                const int sl = need ? suffix_bases(size_t(p), P.dl) : 0;
                const uint32_t seg = uint32_t(__popc(x & ((1u << lane) - 1u)));
                uint32_t tx[2 * W], mask[2 * W];
                suffix_text<W>(a.pk, size_t(p), sl, from, tx, mask);
                // the lane of the longest suffix of this lane's sub-bucket
                const int first = 31 - __clz(((x << 1) | 1u) & (0xffffffffu >> (31 - lane)));
                const int last = lane < len ? lane + __ffs(x >> lane) - 1 : lane;
                unsigned longest = (unsigned(sl) << 5) | unsigned(lane);
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, longest, o);
                    if (lane - o >= first) longest = max(longest, y);
                }
                const int pivot = int(__shfl_sync(0xffffffffu, longest, last) & 31u);
                uint32_t where[2 * W];              // a bit per differing base (its lower one)
                int np = 0;
                #pragma unroll
                for (int i = 0; i < 2 * W; ++i) {
                    const uint32_t y = __shfl_sync(0xffffffffu, tx[i], pivot);
                    const uint32_t d = __reduce_or_sync(0xffffffffu, (tx[i] ^ y) & mask[i]);
                    where[i] = (d | (d >> 1)) & 0x55555555u;
                    np += __popc(where[i]);
                }
                const uint64_t low = (((uint64_t(unsigned(sl)) << P.P) | p) << 5) | uint64_t(unsigned(lane));
                const int low_bits = len_bits + P.P + 5;
                const int seg_bits = 32 - __clz(__popc(x) - 1);
                int src;
                if (np <= 27) {
                    // the bases there, in order, below the sub-bucket's number
                    uint32_t k0 = seg, k1 = 0;
                    #pragma unroll
                    for (int i = 0; i < 2 * W; ++i) {
                        for (uint32_t y = where[i]; y;) {
                            const int z = __clz(y);                     // the base's upper bit is one higher
                            k1 = __funnelshift_l(k0, k1, 2);
                            k0 = __funnelshift_l(tx[i] << (z - 1), k0, 2);
                            y &= 0x7fffffffu >> z;
                        }
                    }
                    const uint64_t k = (uint64_t(k1) << 32) | k0;
                    if (seg_bits + 2 * np + low_bits <= 64) {
                        uint64_t key = lane < len ? (k << low_bits) | low : ~uint64_t(0);
                        warp_sort(key, len, lane);
                        src = int(key & 31u);
                    } else {
                        SortItem<1, uint64_t> it;
                        it.w[0] = lane < len ? k : ~uint64_t(0);
                        it.tail = lane < len ? low : ~uint64_t(0);
                        warp_sort(it, len, lane);
                        src = int(it.tail & 31u);
                    }
                } else {
                    SortItem<W, uint64_t> it;
                    pack_words<W, 5>(tx, seg, it.w);
                    it.tail = low;
                    if (lane >= len) {
                        #pragma unroll
                        for (int j = 0; j < W; ++j) it.w[j] = ~uint64_t(0);
                        it.tail = ~uint64_t(0);
                    }
                    warp_sort(it, len, lane);
                    src = int(it.tail & 31u);
                }
                const uint64_t sorted = __shfl_sync(0xffffffffu, e, src);
                if (lane < len) se[cur + lane] = sorted;
                __syncwarp();
            }
            cur += len;
        }
        __syncthreads();
        // the finished rows
        for (int j = tid; j < m; j += T) {
            const uint64_t e = se[j];
            a.sa[bk.start + j] = idx_t((e >> kSymBits) & pos_mask);
            if (a.bwt) a.bwt[bk.start + j] = uint8_t(e & 7u);
            if (a.kx && !off) a.kx[bk.start + j] = uint16_t((e >> a.kx_shift) & ((1u << a.kx_bits) - 1u));
        }
        if (a.kt && !off) {
            // k-mer of a row (k <= head): the bucket's first d1 bits and the key; absent in a
            // suffix of fewer bases.  Buckets of whole k-mers write each one's two rows; when a
            // k-mer spans buckets its rows are agreed on by minimum and maximum.
            const int k = a.kmer_k, top = 2 * k - P.d1;
            const uint64_t id1 = uint64_t(bk.id_off & ((1u << kIdBits) - 1)) >> P.d2;
            const int low = max(P.key_shift + P.kbits - top, 0);        // lowest k-mer bit of an element
            auto has = [&](uint64_t e) { return int((e >> P.len_shift) & 31u) >= k; };
            const bool spans = a.kmer_spans;
            for (int j = tid; j < m; j += T) {
                const uint64_t e = se[j];
                if (!has(e)) continue;
                bool begins = j == 0, ends = j + 1 == m;
                if (!begins) {
                    const uint64_t y = se[j - 1];
                    begins = (top > 0 && ((e ^ y) >> low)) || !has(y);
                }
                if (!ends) {
                    const uint64_t y = se[j + 1];
                    ends = (top > 0 && ((e ^ y) >> low)) || !has(y);
                }
                if (!begins && !ends) continue;
                const uint64_t key = e >> P.key_shift;
                const size_t c = size_t(top >= 0 ? (id1 << top) | (key >> (P.kbits - top)) : id1 >> (-top));
                const idx_t row = idx_t(a.row0 + bk.start + j);
                if (begins) {
                    if (spans) atomicMin(reinterpret_cast<kmer_int*>(a.kt + 2 * c), kmer_int(row));
                    else a.kt[2 * c] = row;
                }
                if (ends) {
                    if (spans) atomicMax(reinterpret_cast<kmer_int*>(a.kt + 2 * c + 1), kmer_int(row));
                    else a.kt[2 * c + 1] = row;
                }
            }
        }
        __syncthreads();
    }
}

template <int CAP>
static constexpr size_t local_smem() { return size_t(CAP) * 8 + (kLocalBins / 2 + CAP / 32 + 2) * sizeof(unsigned); }

// ------------------------------------------------------------------------------ larger groups
//
// Suffixes equal in all bases of their elements, listed by position: 33..128 are sorted by one warp
// (4 slots a lane, several groups packed and told apart by a segment number), 129..1024 by one CTA
// in shared memory.  A listed group starts at element `start` and is equal up to base `from`.

__device__ __forceinline__ int group_size(unsigned long long g) { return int(g & 0x3fffu); }
__device__ __forceinline__ int group_from(unsigned long long g) { return int((g >> 14) & 0x3ffu); }

constexpr int kRefineThreads = 256;

// BWT symbol of the suffix at p: 0 (`$`) at a read start, else the preceding base (1..4)
__device__ __forceinline__ uint8_t bwt_symbol(const uint64_t* __restrict__ pk, size_t p, const DivL& dl) {
    if (suffix_bases(p, dl) == int(dl.L)) return 0;
    const size_t q = p - 1;
    return uint8_t(((pk[q >> 5] >> (62 - 2 * int(q & 31))) & 3) + 1);
}

// The warp's 128 slots (slot e * 32 + lane is register set e of that lane) take consecutive listed
// groups while they fit; one bitonic network on (segment, bases from `from` on, length, slot)
// sorts every packed group in place.  A group's members arrive in ascending position, so the slot
// breaks ties exactly as the position does; positions and symbols wait in shared memory and are
// gathered by slot at the end.  Distances below 32 exchange by shuffle, larger ones swap
// registers within a lane.
template <int W>
__global__ void __launch_bounds__(kRefineThreads, W <= 4 ? 3 : 1)
k_refine_warp(const unsigned long long* __restrict__ list, const unsigned long long* __restrict__ cnt,
              const uint64_t* __restrict__ pk, DivL dl, idx_t* __restrict__ val, uint8_t* __restrict__ bwt) {
    constexpr int kChunk = 8, E = 4, N = 32 * E;
    __shared__ idx_t spos[kRefineThreads / 32][N];
    __shared__ uint8_t ssym[kRefineThreads / 32][N];
    const int lane = threadIdx.x & 31;
    idx_t* const mypos = spos[threadIdx.x >> 5];
    uint8_t* const mysym = ssym[threadIdx.x >> 5];
    const size_t warp = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const size_t nwarps = (size_t(gridDim.x) * blockDim.x) >> 5;
    const size_t groups = *cnt;
    for (size_t c0 = warp * kChunk; c0 < groups; c0 += nwarps * kChunk) {
        const unsigned long long mine = (lane < kChunk && c0 + lane < groups) ? list[c0 + lane] : 0ull;
        int next = 0;
        while (next < kChunk) {
            // consecutive entries next .. next + taken - 1 fit in N slots
            int taken = 0, total = 0;
            uint32_t seg[E];
            size_t at[E];
            int from[E];
            #pragma unroll
            for (int e = 0; e < E; ++e) {
                seg[e] = 255;
                at[e] = 0;
                from[e] = 0;
            }
            for (int q = next; q < kChunk; ++q) {
                const unsigned long long x = __shfl_sync(0xffffffffu, mine, q);
                const int m = group_size(x);
                if (m == 0 || total + m > N) break;
                #pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int slot = e * 32 + lane;
                    if (slot >= total && slot < total + m) {
                        seg[e] = uint32_t(q - next);
                        at[e] = size_t(x >> 24) + size_t(slot - total);
                        from[e] = group_from(x);
                    }
                }
                total += m;
                ++taken;
            }
            if (taken == 0) break;
            SortItem<W, uint32_t> it[E];
            #pragma unroll
            for (int e = 0; e < E; ++e) {
                if (seg[e] != 255) {
                    const idx_t pos = val[at[e]];
                    const int len = suffix_bases(size_t(pos), dl);
                    sort_words<W, 3>(pk, size_t(pos), len, from[e], seg[e], it[e].w);
                    it[e].tail = (uint32_t(len) << 8) | uint32_t(e * 32 + lane);
                    mypos[e * 32 + lane] = pos;
                    if (bwt) mysym[e * 32 + lane] = bwt_symbol(pk, size_t(pos), dl);
                } else {
                    #pragma unroll
                    for (int j = 0; j < W; ++j) it[e].w[j] = ~uint64_t(0);
                    it[e].tail = ~0u;
                }
            }
            #pragma unroll
            for (int k = 2; k <= N; k <<= 1) {
                #pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    if (j >= 32) {
                        #pragma unroll
                        for (int e = 0; e < E; ++e) {
                            const int f = e ^ (j >> 5);
                            if (f > e) {
                                const bool asc = ((e * 32 + lane) & k) == 0;
                                if (item_less<W>(it[f], it[e]) == asc) {
                                    const SortItem<W, uint32_t> t = it[e];
                                    it[e] = it[f];
                                    it[f] = t;
                                }
                            }
                        }
                    } else {
                        #pragma unroll
                        for (int e = 0; e < E; ++e) {
                            SortItem<W, uint32_t> o;
                            #pragma unroll
                            for (int q = 0; q < W; ++q) o.w[q] = __shfl_xor_sync(0xffffffffu, it[e].w[q], j);
                            o.tail = __shfl_xor_sync(0xffffffffu, it[e].tail, j);
                            const bool keep_min = ((lane & j) == 0) == (((e * 32 + lane) & k) == 0);
                            if (keep_min == item_less<W>(o, it[e])) it[e] = o;
                        }
                    }
                }
            }
            __syncwarp();
            #pragma unroll
            for (int e = 0; e < E; ++e) {
                if (seg[e] != 255) {
                    val[at[e]] = mypos[it[e].tail & 255u];
                    if (bwt) bwt[at[e]] = mysym[it[e].tail & 255u];
                }
            }
            __syncwarp();
            next += taken;
        }
    }
}

// the (words, length, position) order of two suffixes
template <int W>
__device__ __forceinline__ bool tuple_less(const uint64_t a[W], uint64_t alen, uint64_t apos, const uint64_t b[W],
                                           uint64_t blen, uint64_t bpos) {
    #pragma unroll
    for (int j = 0; j < W; ++j)
        if (a[j] != b[j]) return a[j] < b[j];
    if (alen != blen) return alen < blen;
    return apos < bpos;
}

// one CTA's bitonic sort of one group of m suffixes held as columns: words w[j][m], len[m], pos[m];
// comparators all point up (a mirrored first step per merge), so that places past m are skipped
template <int W>
__device__ void cta_bitonic(uint64_t* cols, int m) {
    uint64_t* lenc = cols + size_t(W) * m;
    uint64_t* posc = lenc + m;
    auto exchange = [&](int i, int o) {
        if (o >= m) return;
        uint64_t a[W], b[W];
        #pragma unroll
        for (int q = 0; q < W; ++q) {
            a[q] = cols[size_t(q) * m + i];
            b[q] = cols[size_t(q) * m + o];
        }
        const uint64_t al = lenc[i], ap = posc[i], bl = lenc[o], bp = posc[o];
        if (!tuple_less<W>(b, bl, bp, a, al, ap)) return;
        #pragma unroll
        for (int q = 0; q < W; ++q) {
            cols[size_t(q) * m + i] = b[q];
            cols[size_t(q) * m + o] = a[q];
        }
        lenc[i] = bl;
        posc[i] = bp;
        lenc[o] = al;
        posc[o] = ap;
    };
    for (int k = 2; k < 2 * m; k <<= 1) {
        const int half = k >> 1, pairs = (m + k - 1) / k * half;
        for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
            const int q = i / half, o = i - q * half;
            exchange(q * k + o, q * k + k - 1 - o);
        }
        __syncthreads();
        for (int j = half >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
                const int a = ((i & ~(j - 1)) << 1) | (i & (j - 1));
                exchange(a, a + j);
            }
            __syncthreads();
        }
    }
}

template <int W>
__device__ void cta_load_group(uint64_t* cols, size_t start, int m, const uint64_t* __restrict__ pk, const DivL& dl,
                               const idx_t* __restrict__ val, int off) {
    uint64_t* lenc = cols + size_t(W) * m;
    uint64_t* posc = lenc + m;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        uint64_t w[W];
        const uint64_t pos = uint64_t(val[start + i]), len = uint64_t(suffix_bases(size_t(pos), dl));
        sort_words<W, 0>(pk, size_t(pos), int(len), off, 0, w);
        #pragma unroll
        for (int q = 0; q < W; ++q) cols[size_t(q) * m + i] = w[q];
        lenc[i] = len;
        posc[i] = pos;
    }
    __syncthreads();
}

template <int W>
__global__ void k_refine_cta(const unsigned long long* __restrict__ list, const unsigned long long* __restrict__ cnt,
                             const uint64_t* __restrict__ pk, DivL dl, idx_t* __restrict__ val, uint8_t* __restrict__ bwt) {
    extern __shared__ uint64_t s_cols[];
    const size_t groups = *cnt;
    for (size_t g = blockIdx.x; g < groups; g += gridDim.x) {
        const unsigned long long e = list[g];
        const size_t start = size_t(e >> 24);
        const int m = group_size(e);
        cta_load_group<W>(s_cols, start, m, pk, dl, val, group_from(e));
        cta_bitonic<W>(s_cols, m);
        const uint64_t* posc = s_cols + size_t(W + 1) * m;
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const idx_t pos = idx_t(posc[i]);
            val[start + i] = pos;
            if (bwt) bwt[start + i] = bwt_symbol(pk, size_t(pos), dl);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------ further splits
//
// Buckets of more than kLocalLarge suffixes and groups of more than 1024 suffixes equal in all bases
// of their elements (low-complexity or highly repeated sequence), driven by the host: a range is
// split by the 10 highest bits in which its elements differ -- text, else length, else, among equal
// strings, position -- and one whose suffixes all go on past equal heads first gets new elements
// of its next bases, until every part fits the local kernel.

constexpr int kMoreRanges = 4096;           // ranges described at a time
constexpr int kMoreMerge = 2048;            // children put together for the local kernel
// ranges split at a time (16 KB each: a quarter byte a suffix)
static size_t more_splits_at(size_t m) { return std::min<size_t>(1024, std::max<size_t>(64, m >> 16)); }

// new elements for ranges whose suffixes are equal in their first off[range] bases: the next
// more_bits / 2 of them, left-aligned in the key
__global__ void __launch_bounds__(kSplitThreads) k_more_rebuild(const uint64_t* __restrict__ pk, MsdPlan a, int more_bits,
                                                                MsdRanges r, const int* __restrict__ off,
                                                                uint64_t* __restrict__ buf) {
    const unsigned tiles = r.tile0[r.count];
    for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int q = range_of(r, t);
        const size_t b = r.start[q] + size_t(t - r.tile0[q]) * kSplitTile;
        const size_t e = zmin(r.end[q], b + kSplitTile);
        for (size_t i = b + threadIdx.x; i < e; i += kSplitThreads) {
            const uint64_t low = buf[i] & ((uint64_t(1) << a.len_shift) - 1);
            const size_t p = size_t(low >> kSymBits);
            const int rem = suffix_bases(p, a.dl) - off[q];
            uint64_t key = 0;
            int w = 0;
            if (rem > 0) {
                uint64_t x = window(pk, p + size_t(off[q]));
                if (rem < 32) x &= ~uint64_t(0) << (64 - 2 * rem);
                key = (x >> (64 - more_bits)) << (a.kbits - more_bits);
                w = rem < more_bits / 2 ? rem : more_bits / 2;
            }
            buf[i] = (key << a.key_shift) | (uint64_t(w) << a.len_shift) | low;
        }
    }
}

// the bits in which each range's elements differ, and its first element
__global__ void __launch_bounds__(kSplitThreads) k_more_diff(const uint64_t* __restrict__ buf, MsdRanges r,
                                                             unsigned long long* __restrict__ diff,
                                                             unsigned long long* __restrict__ e0) {
    const unsigned tiles = r.tile0[r.count];
    for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int q = range_of(r, t);
        const size_t b = r.start[q] + size_t(t - r.tile0[q]) * kSplitTile;
        const size_t e = zmin(r.end[q], b + kSplitTile);
        const uint64_t first = buf[r.start[q]];
        uint64_t d = 0;
        for (size_t i = b + threadIdx.x; i < e; i += kSplitThreads) d |= buf[i] ^ first;
        const unsigned lo = __reduce_or_sync(0xffffffffu, unsigned(d)), hi = __reduce_or_sync(0xffffffffu, unsigned(d >> 32));
        if ((threadIdx.x & 31) == 0) atomicOr(&diff[q], (unsigned long long)((uint64_t(hi) << 32) | lo));
        if (threadIdx.x == 0 && b == r.start[q]) e0[q] = first;
    }
}

// The children of range blockIdx.x from their counts: their places (cursor, which the split advances) and,
// from large[listed] on, their buckets.  Neighbours are one where they start in the same kMoreMerge elements
// of the range (ten thousand equal strings split by position would else be a thousand buckets: 10 K equal
// reads of 100 bases 5.3 ms, 2.3 together); children of more than kLocalLarge go to `again`, the first of
// them also to r.first.  Listed here, their counts stay on the device: at 20 % GC half of 143 M suffixes come
// in 3.4 thousand buckets that have to be split.  With 8 KB of counts of each read by the host, and two
// launches for the k-mers of each, an index of both directions took 107 ms (radix passes and refinement
// 26), now 18.8.
struct MoreLists {
    unsigned long long large, more;         // listed in `large` and in `again`
    MsdBucket first[256];
};
__global__ void __launch_bounds__(kScanThreads) k_more_list(const unsigned long long* __restrict__ cnt, MsdRanges r,
                                                            const int* __restrict__ off, unsigned long long* __restrict__ cursor,
                                                            unsigned listed, MsdBucket* __restrict__ large, unsigned cap_large,
                                                            MsdBucket* __restrict__ again, unsigned cap_again,
                                                            MoreLists* __restrict__ c) {
    constexpr int kBins = 1 << kMoreBits, kPer = kBins / kScanThreads, kWords = kBins / 32;
    __shared__ unsigned pref[kBins], wsum[kScanThreads / 32], some[kWords], begin[kWords];
    __shared__ unsigned long long wtot;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned long long* const n = cnt + (size_t(blockIdx.x) << kMoreBits);
    const unsigned long long start = r.start[blockIdx.x];
    const unsigned id_off = (unsigned(off[blockIdx.x]) << kIdBits) | (unsigned(r.shift[blockIdx.x]) >> 6);
    if (tid < kWords) some[tid] = begin[tid] = 0;
    unsigned v[kPer], mine = 0;                 // (a range has fewer than 2^32 elements)
    #pragma unroll
    for (int i = 0; i < kPer; ++i) mine += v[i] = unsigned(n[tid * kPer + i]);
    unsigned x = mine;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned run = x - mine;
    for (int w = 0; w < warp; ++w) run += wsum[w];
    #pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int b = tid * kPer + i;
        pref[b] = run;
        cursor[(size_t(blockIdx.x) << kMoreBits) + b] = start + run;
        if (v[i]) atomicOr(&some[b >> 5], 1u << (b & 31));
        run += v[i];
    }
    if (tid == kScanThreads - 1) wtot = run;
    __syncthreads();
    // the first child from b + 1 on in a mask, or kBins
    auto next = [](const unsigned* mask, int b) {
        for (int w = (b + 1) >> 5; w < kWords; ++w) {
            const unsigned y = w == (b + 1) >> 5 ? mask[w] & (~0u << ((b + 1) & 31)) : mask[w];
            if (y) return 32 * w + __ffs(y) - 1;
        }
        return kBins;
    };
    // where a bucket begins: at a child too large for company, after one, and where another kMoreMerge begins
    #pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int b = tid * kPer + i;
        if (!v[i]) continue;
        const bool alone = v[i] > unsigned(kLocalLarge - kMoreMerge);
        if (alone || pref[b] == 0) atomicOr(&begin[b >> 5], 1u << (b & 31));
        if (alone || pref[b] / kMoreMerge != (pref[b] + v[i]) / kMoreMerge) {
            const int e = next(some, b);
            if (e < kBins) atomicOr(&begin[e >> 5], 1u << (e & 31));
        }
    }
    __syncthreads();
    #pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int b = tid * kPer + i;
        if (!((begin[b >> 5] >> (b & 31)) & 1u)) continue;
        const int e = next(begin, b);
        const unsigned size = (e < kBins ? pref[e] : unsigned(wtot)) - pref[b];
        const bool fits = size <= unsigned(kLocalLarge);
        const MsdBucket bucket{start + pref[b], size, id_off};
        const unsigned long long at = fits ? listed + atomicAdd(&c->large, 1ull) : atomicAdd(&c->more, 1ull);
        if (at < (fits ? cap_large : cap_again)) (fits ? large : again)[at] = bucket;
        if (!fits && at < sizeof c->first / sizeof c->first[0]) c->first[at] = bucket;
    }
}

__global__ void __launch_bounds__(kSplitThreads) k_more_copy(const uint64_t* __restrict__ from, MsdRanges r,
                                                             uint64_t* __restrict__ to) {
    const unsigned tiles = r.tile0[r.count];
    for (unsigned t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int q = range_of(r, t);
        const size_t b = r.start[q] + size_t(t - r.tile0[q]) * kSplitTile;
        const size_t e = zmin(r.end[q], b + kSplitTile);
        for (size_t i = b + threadIdx.x; i < e; i += kSplitThreads) to[i] = from[i];
    }
}

// A k-mer table whose k-mers span buckets is entered by minimum and maximum: prepared so (mode 0;
// mode 2 only where a k-mer is still absent), then absent ones set as everywhere else (mode 1:
// last < first).  Of all k-mers, or of those of `count` listed buckets, 2^shift each.
__global__ void k_kmer_span(idx_t* __restrict__ kt, size_t count, int mode, const MsdBucket* __restrict__ list, int shift) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t j = size_t(blockIdx.x) * blockDim.x + threadIdx.x; j < count << shift; j += stride) {
        size_t i = j;
        if (list) i = (size_t(list[j >> shift].id_off & ((1u << kIdBits) - 1)) << shift) | (j & ((size_t(1) << shift) - 1));
        idx_t* const k = kt + 2 * i;
        if (mode == 0 || (mode == 2 && k[1] < k[0])) {
            k[0] = ~idx_t(0);
            k[1] = 0;
        } else if (mode == 1 && k[0] == ~idx_t(0)) {
            k[0] = 1;
        }
    }
}

// rows [r0, r1) all start with k-mer c
__global__ void k_kmer_rows(idx_t* __restrict__ kt, size_t c, size_t r0, size_t r1) {
    atomicMin(reinterpret_cast<kmer_int*>(kt + 2 * c), kmer_int(r0));
    atomicMax(reinterpret_cast<kmer_int*>(kt + 2 * c + 1), kmer_int(r1 - 1));
}
// and go on with the same bases
__global__ void k_kx_rows(uint16_t* __restrict__ kx, size_t m, uint16_t v) {
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m; i += stride) kx[i] = v;
}

// ------------------------------------------------------------------------------ driver

static size_t al(size_t b) { return (b + 255) & ~size_t(255); }

namespace {

// The working memory of one sort of `m` suffixes at a time out of n.
struct MsdScratch {
    uint64_t *a, *b;                                // elements after the first and the second pass
    unsigned long long *hist, *cnt, *shorts;        // cleared together with the counters
    MsdCounters* counters;
    size_t clear_bytes;
    unsigned long long *start1, *cursor1, *lstart, *cursor, *sfirst;
    unsigned* tile0;
    MsdBucket *small, *large, *more;
    unsigned long long *mid, *big, *huge;
    size_t cap_list, cap_more, cap_mid, cap_big, cap_huge;
    uint32_t *sk0, *sk1;                            // short suffixes
    idx_t *sv0, *sv1;
    void* rtmp;
    size_t rtmp_bytes;
    unsigned char* r_desc;                          // further splits: a RangeBlock,
    unsigned long long *r_diff, *r_cnt, *r_cursor;  // r_diff: differences, then first elements
    MoreLists* r_lists;                             // before r_cnt, cleared with it
    MsdBucket* again;
    size_t splits;
    uint64_t* pk;
    uint8_t* bwt;
    unsigned long long* hist6;
    size_t bytes;
};

MsdScratch msd_layout(void* base, const MsdPlan& p, size_t m, size_t nr) {
    MsdScratch s{};
    size_t used = 0;
    auto take = [&](size_t bytes) {
        char* q = base ? static_cast<char*>(base) + used : nullptr;
        used += al(bytes);
        return q;
    };
    using U = unsigned long long;
    const size_t bins1 = size_t(1) << p.d1, buckets = size_t(1) << (p.d1 + p.d2);
    const bool two = p.d2 > 0;
    // 64-bit suffix arrays hold the first pass's elements themselves
    s.a = sizeof(idx_t) == 4 ? reinterpret_cast<uint64_t*>(take(m * 8)) : nullptr;
    s.b = reinterpret_cast<uint64_t*>(take(m * 8));
    const size_t z0 = used;
    s.counters = reinterpret_cast<MsdCounters*>(take(sizeof(MsdCounters)));
    s.hist = reinterpret_cast<U*>(take(bins1 * 8));
    s.cnt = reinterpret_cast<U*>(take(two ? buckets * 8 : 0));
    s.shorts = reinterpret_cast<U*>(take(p.S ? buckets * 8 : 0));
    s.clear_bytes = used - z0;
    s.sfirst = reinterpret_cast<U*>(take(p.S ? buckets * 8 : 0));
    s.start1 = reinterpret_cast<U*>(take(bins1 * 8));
    s.cursor1 = reinterpret_cast<U*>(take(bins1 * 8));
    s.tile0 = reinterpret_cast<unsigned*>(take((bins1 + 1) * 4));
    s.lstart = reinterpret_cast<U*>(take(buckets * 8));
    s.cursor = reinterpret_cast<U*>(take(buckets * 8));
    s.cap_list = std::max<size_t>(buckets, kMoreRanges);
    s.small = reinterpret_cast<MsdBucket*>(take(buckets * sizeof(MsdBucket)));
    s.large = reinterpret_cast<MsdBucket*>(take(s.cap_list * sizeof(MsdBucket)));
    s.cap_more = m / (kLocalLarge + 1) + 1;
    s.cap_mid = m / 33 + 1;
    s.cap_big = m / 129 + 1;
    s.cap_huge = m / 1025 + 1;
    s.more = reinterpret_cast<MsdBucket*>(take(s.cap_more * sizeof(MsdBucket)));
    s.mid = reinterpret_cast<U*>(take(s.cap_mid * 8));
    s.big = reinterpret_cast<U*>(take(s.cap_big * 8));
    s.huge = reinterpret_cast<U*>(take(s.cap_huge * 8));
    const size_t sh = nr * size_t(p.S);
    s.sk0 = reinterpret_cast<uint32_t*>(take(sh * 4));
    s.sk1 = reinterpret_cast<uint32_t*>(take(sh * 4));
    s.sv0 = reinterpret_cast<idx_t*>(take(sh * sizeof(idx_t)));
    s.sv1 = reinterpret_cast<idx_t*>(take(sh * sizeof(idx_t)));
    s.rtmp_bytes = p.S ? radix_tmp_bytes(sh) : 0;
    s.rtmp = take(s.rtmp_bytes);
    s.r_desc = reinterpret_cast<unsigned char*>(take(RangeBlock{size_t(kMoreRanges)}.bytes()));
    s.r_diff = reinterpret_cast<U*>(take(2 * kMoreRanges * 8));
    s.splits = more_splits_at(m);
    s.r_lists = reinterpret_cast<MoreLists*>(take(sizeof(MoreLists)));
    s.r_cnt = reinterpret_cast<U*>(take((s.splits << kMoreBits) * 8));
    s.r_cursor = reinterpret_cast<U*>(take((s.splits << kMoreBits) * 8));
    s.again = reinterpret_cast<MsdBucket*>(take(s.cap_more * sizeof(MsdBucket)));
    s.pk = reinterpret_cast<uint64_t*>(take((p.n / 32 + 4) * 8));
    s.bwt = reinterpret_cast<uint8_t*>(take(p.n));
    s.hist6 = reinterpret_cast<U*>(take(size_t(kBuckets) * 8));
    s.bytes = used;
    return s;
}

// Working memory of prefix doubling: two 64-bit key arrays, one value array (the other is the
// suffix array), 32-bit ranks, packed text, per-tile group heads.
size_t doubling_bytes(size_t n) {
    const size_t tiles = (n + HT_TILE - 1) / HT_TILE + 1;
    return 2 * al(n * sizeof(uint64_t)) + al(n * sizeof(idx_t)) + al(n * sizeof(uint32_t)) +
           al((n / 32 + 4) * sizeof(uint64_t)) + al(radix_tmp_bytes(n)) + al(3 * tiles * sizeof(unsigned long long)) +
           1024;
}

// What a sort in chunks of `cap` suffixes may take: 20 bytes and two positions a suffix of a chunk
// and 3 1/4 bytes a suffix of the index.  One pass over everything is used when it needs no more.
size_t chunk_budget(size_t n, size_t cap) { return cap * (20 + 2 * sizeof(idx_t)) + 3 * n + n / 4; }

struct SortShape {
    MsdPlan plan;
    bool doubling, chunked;
    size_t m;               // suffixes sorted at a time
    size_t bytes;
};

SortShape sort_shape(size_t n, size_t nr, int L, size_t cap) {
    SortShape s{};
    s.plan = make_plan(n, nr, idx_t(L), true, false);
    s.m = n;
    if (plan_words(s.plan) > kMaxWords) {
        s.doubling = true;
        s.bytes = doubling_bytes(n);
        return s;
    }
    s.bytes = msd_layout(nullptr, s.plan, n, nr).bytes + 1024;
    if (cap && cap < n && s.bytes > chunk_budget(n, cap)) {
        s.chunked = true;
        s.m = cap;
        for (bool shorts : {true, false}) {             // short suffixes apart where there is room for them
            s.plan = make_plan(n, nr, idx_t(L), shorts && n >= (size_t(1) << 22), true);
            s.bytes = msd_layout(nullptr, s.plan, cap, nr).bytes + 1024;
            if (s.bytes <= chunk_budget(n, cap)) break;
        }
    }
    return s;
}

struct SortRange {
    unsigned long long start, end;
    int off;
    unsigned id;            // off = 0: the bucket it is part of
    bool rebuild;
};

template <int W>
struct MsdKernels {
    static int local_blocks(bool large, int sms) {
        static_assert(W >= 1 && W <= kMaxWords, "networks of 1 .. kMaxWords words");
        int per = 0;
        const cudaError_t e = large
            ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_msd_local<W, kLocalLarge, 256>, 256, local_smem<kLocalLarge>())
            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_msd_local<W, kLocalSmall, 128>, 128, local_smem<kLocalSmall>());
        if (e != cudaSuccess) cudaGetLastError();
        return (e == cudaSuccess && per > 0 ? per : 1) * sms;
    }
    static constexpr size_t kCtaSmem = size_t(W + 2) * 1024 * sizeof(uint64_t);
    static cudaError_t prepare() {
        cudaError_t e = allow_smem<local_smem<kLocalSmall>()>(k_msd_local<W, kLocalSmall, 128>);
        if (e == cudaSuccess) e = allow_smem<local_smem<kLocalLarge>()>(k_msd_local<W, kLocalLarge, 256>);
        if (e == cudaSuccess) e = allow_smem<kCtaSmem>(k_refine_cta<W>);
        if (e == cudaSuccess) e = allow_smem<MsdSmem::bytes(kMaxDigit, true)>(k_msd_text<uint64_t>);
        if (e == cudaSuccess) e = allow_smem<MsdSmem::bytes(kMaxDigit, true)>(k_msd_text<uint32_t>);
        if (e == cudaSuccess) e = allow_smem<MsdSmem::bytes(kMaxDigit, false)>(k_msd_split);
        return e;
    }
    static void local(bool large, MsdLocal a, const MsdScratch& s, size_t most, int sms, cudaStream_t st) {
        a.list = large ? s.large : s.small;
        a.count = large ? &s.counters->large : &s.counters->small;
        a.next = large ? &s.counters->next_large : &s.counters->next_small;
        const unsigned g = unsigned(std::max<size_t>(1, std::min<size_t>(most, size_t(local_blocks(large, sms)))));
        if (large) k_msd_local<W, kLocalLarge, 256><<<g, 256, local_smem<kLocalLarge>(), st>>>(a);
        else k_msd_local<W, kLocalSmall, 128><<<g, 128, local_smem<kLocalSmall>(), st>>>(a);
        note_launch();
    }
    static void groups(const MsdLocal& a, const MsdScratch& s, int sms, cudaStream_t st) {
        const size_t warps = (s.cap_mid + 7) / 8;
        const unsigned g = unsigned(std::max<size_t>(1, std::min<size_t>((warps + 7) / 8, size_t(sms) * 4)));
        k_refine_warp<W><<<g, kRefineThreads, 0, st>>>(s.mid, &s.counters->mid, a.pk, a.plan.dl, a.sa, a.bwt);
        note_launch();
        k_refine_cta<W><<<unsigned(std::min<size_t>(s.cap_big, size_t(sms) * 2)), 512, kCtaSmem, st>>>(
            s.big, &s.counters->big, a.pk, a.plan.dl, a.sa, a.bwt);
        note_launch();
    }
};

// The further splits (see above) of the listed buckets and groups.
template <int W>
int more_splits(const MsdCounters& c0, MsdLocal a, const MsdScratch& s, uint64_t* tmp, int sms, cudaStream_t st) {
    const MsdPlan& P = a.plan;
    const int k = a.kmer_k, bits = P.d1 + P.d2;
    const bool own_span = a.kt && !a.kmer_spans;        // a listed bucket's k-mers span its parts
    auto wait_stream = [st] { return cudaStreamSynchronize(st); };
    HeldBlocks<decltype(wait_stream)> held(wait_stream);        // the sources of copies to the device
    auto h2d = [&](void* d, const void* h, size_t b) {
        return cudaMemcpyAsync(d, std::memcpy(held.take(b), h, b), b, cudaMemcpyHostToDevice, st);
    };
    auto d2h = [&](void* h, const void* d, size_t b) { return cudaMemcpyAsync(h, d, b, cudaMemcpyDeviceToHost, st); };
    std::vector<SortRange> work;
    auto take_huge = [&](unsigned long long count) -> int {
        if (count > s.cap_huge) return int(cudaErrorUnknown);
        std::vector<unsigned long long> h(count);
        if (count) d2h(h.data(), s.huge, count * 8);
        const cudaError_t e = held.wait();
        if (e != cudaSuccess) return int(e);
        for (unsigned long long g : h)
            work.push_back({g >> 24, (g >> 24) + (g & 0x3fff), int((g >> 14) & 0x3ff), 0, true});
        return 0;
    };
    {
        if (c0.more > s.cap_more) return int(cudaErrorUnknown);
        std::vector<MsdBucket> m(c0.more);
        if (c0.more) d2h(m.data(), s.more, c0.more * sizeof(MsdBucket));
        const int rc = take_huge(c0.huge);
        if (rc) return rc;
        for (const MsdBucket& b : m) {
            if (b.size == 0xffffffffu) return int(cudaErrorInvalidValue);       // 2^32 and more in one bucket
            const unsigned id = b.id_off & ((1u << kIdBits) - 1);
            work.push_back({b.start, b.start + b.size, 0, id, false});
        }
    }
    const int per = 2 * k - bits;                       // s.more keeps the listed buckets, whose k-mers are 2^per each
    auto span = [&](int mode) {
        k_kmer_span<<<grid_for(size_t(c0.more) << per, 256), 256, 0, st>>>(a.kt, size_t(c0.more), mode, s.more, per);
        note_launch();
    };
    if (own_span && c0.more) span(2);
    if (own_span) a.kmer_spans = 1;
    // the buckets of s.large finished; their groups of more than 1024 come back
    size_t listed = 0;
    auto finish = [&]() -> int {
        MsdCounters c{};
        c.large = listed;
        h2d(s.counters, &c, sizeof c);
        MsdKernels<W>::local(true, a, s, listed, sms, st);
        MsdKernels<W>::groups(a, s, sms, st);
        d2h(&c, s.counters, sizeof c);
        const cudaError_t e = held.wait();
        if (e != cudaSuccess) return int(e);
        listed = 0;
        if (c.mid > s.cap_mid || c.big > s.cap_big) return int(cudaErrorUnknown);
        return take_huge(c.huge);
    };
    // describes ranges v[i0, i1) (at most kMoreRanges) and their shifts on the device, one copy for all
    unsigned tiles = 0;
    const int* r_off = nullptr;
    auto describe = [&](const std::vector<SortRange>& v, size_t i0, size_t i1, const int* shift) {
        const RangeBlock b{i1 - i0};
        unsigned char* const h = held.take(b.bytes());
        tiles = fill_ranges(h, v.data() + i0, i1 - i0, shift, size_t(kSplitTile));
        cudaMemcpyAsync(s.r_desc, h, b.bytes(), cudaMemcpyHostToDevice, st);
        r_off = reinterpret_cast<const int*>(s.r_desc + b.offs());
        MsdRanges r{};
        r.start = reinterpret_cast<const unsigned long long*>(s.r_desc);
        r.end = reinterpret_cast<const unsigned long long*>(s.r_desc + b.ends());
        r.tile0 = reinterpret_cast<const unsigned*>(s.r_desc + b.tiles());
        r.shift = shift ? reinterpret_cast<const int*>(s.r_desc + b.shifts()) : nullptr;
        r.count = int(i1 - i0);
        return r;
    };
    auto grid = [&] { return std::min(tiles, unsigned(sms * 4)); };
    while (!work.empty() || listed) {
        if (work.empty()) {
            if (const int rc = finish()) return rc;
            continue;
        }
        // new elements where a range's are used up
        std::vector<SortRange> v, fits;
        for (SortRange& r : work)
            if (r.rebuild) v.push_back(r);
        for (size_t i = 0; i < v.size(); i += kMoreRanges) {
            const MsdRanges r = describe(v, i, std::min(v.size(), i + kMoreRanges), nullptr);
            k_more_rebuild<<<grid(), kSplitThreads, 0, st>>>(a.pk, P, a.more_bits, r, r_off, a.buf);
            note_launch();
        }
        v.clear();
        for (SortRange& r : work) {
            r.rebuild = false;
            (r.end - r.start <= size_t(kLocalLarge) ? fits : v).push_back(r);
        }
        work.clear();
        for (size_t i = 0, i1; i < fits.size(); i = i1) {
            if (listed == s.cap_list)
                if (const int rc = finish()) return rc;
            i1 = std::min(fits.size(), i + s.cap_list - listed);
            std::vector<MsdBucket> b;
            for (size_t q = i; q < i1; ++q) b.push_back({fits[q].start, unsigned(fits[q].end - fits[q].start), (unsigned(fits[q].off) << kIdBits) | (fits[q].off ? 0u : fits[q].id)});
            h2d(s.large + listed, b.data(), b.size() * sizeof(MsdBucket));
            listed += b.size();
        }
        // where the others' elements differ
        std::vector<SortRange> split;
        std::vector<int> shift;
        for (size_t i = 0; i < v.size(); i += kMoreRanges) {
            const size_t i1 = std::min(v.size(), i + kMoreRanges);
            const MsdRanges r = describe(v, i, i1, nullptr);
            cudaMemsetAsync(s.r_diff, 0, r.count * 8, st);
            k_more_diff<<<grid(), kSplitThreads, 0, st>>>(a.buf, r, s.r_diff, s.r_diff + r.count);
            note_launch();
            std::vector<unsigned long long> d(2 * size_t(r.count));
            d2h(d.data(), s.r_diff, d.size() * 8);
            const unsigned long long* const e0 = d.data() + r.count;
            const cudaError_t e = held.wait();
            if (e != cudaSuccess) return int(e);
            for (int q = 0; q < r.count; ++q) {
                SortRange x = v[i + q];
                int hb = 63;
                while (hb > 0 && !((d[q] >> hb) & 1)) --hb;
                const int full = x.off ? a.more_bits / 2 : P.head;
                if (hb < P.len_shift && int((e0[q] >> P.len_shift) & 31) == full) {
                    if (a.kt && !x.off) {                // one k-mer throughout
                        const int top = 2 * k - P.d1;
                        const uint64_t id1 = x.id >> P.d2, key = e0[q] >> P.key_shift;
                        const uint64_t c = top >= 0 ? (id1 << top) | (key >> (P.kbits - top)) : id1 >> (-top);
                        k_kmer_rows<<<1, 1, 0, st>>>(a.kt, size_t(c), a.row0 + x.start, a.row0 + x.end);
                        note_launch();
                        if (a.kx) {
                            const size_t m = size_t(x.end - x.start);
                            k_kx_rows<<<grid_for(m, 256), 256, 0, st>>>(
                                a.kx + x.start, m, uint16_t((e0[q] >> a.kx_shift) & ((1u << a.kx_bits) - 1u)));
                            note_launch();
                        }
                    }
                    x.off += full;
                    x.rebuild = true;
                    work.push_back(x);
                    continue;
                }
                int sh = hb - (kMoreBits - 1);
                if (hb >= P.key_shift) sh = std::max(sh, P.key_shift);
                else if (hb >= P.len_shift) sh = P.len_shift;
                split.push_back(x);
                shift.push_back(std::max(sh, 0) | int((x.off ? 0u : x.id) << 6));
            }
        }
        // split, their children's places and buckets from the counts on the device: as many ranges at a
        // time as there is room for their counts and, at most, for their buckets
        for (size_t i = 0, i1; i < split.size(); i = i1) {
            size_t most = listed;
            for (i1 = i; i1 < split.size() && i1 - i < s.splits; ++i1) {
                const size_t n = size_t(split[i1].end - split[i1].start);
                const size_t b = std::min(size_t(1) << kMoreBits, n / kMoreMerge + 2 * (n / (kLocalLarge - kMoreMerge)) + 2);
                if (most + b > s.cap_list) break;
                most += b;
            }
            if (i1 == i) {
                if (const int rc = finish()) return rc;
                continue;
            }
            MsdRanges r = describe(split, i, i1, shift.data() + i);
            r.bits = kMoreBits;
            cudaMemsetAsync(s.r_lists, 0, al(sizeof(MoreLists)) + ((i1 - i) << kMoreBits) * 8, st);
            k_msd_count<<<grid(), kSplitThreads, 0, st>>>(a.buf, r, s.r_cnt);
            k_more_list<<<unsigned(i1 - i), kScanThreads, 0, st>>>(s.r_cnt, r, r_off, s.r_cursor, unsigned(listed), s.large,
                                                                  unsigned(s.cap_list), s.again, unsigned(s.cap_more), s.r_lists);
            k_msd_split<<<grid(), kSplitThreads, MsdSmem::bytes(kMoreBits, false), st>>>(a.buf, r, s.r_cursor, tmp);
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) {
                held.wait();
                return int(e);
            }
            k_more_copy<<<grid(), kSplitThreads, 0, st>>>(tmp, r, a.buf);
            for (int q = 0; q < 4; ++q) note_launch();
            MoreLists c;
            d2h(&c, s.r_lists, sizeof c);
            e = held.wait();
            if (e != cudaSuccess) return int(e);
            if (listed + c.large > s.cap_list || c.more > s.cap_more) return int(cudaErrorUnknown);
            listed += size_t(c.large);
            std::vector<MsdBucket> again(c.first, c.first + std::min<size_t>(c.more, 256));
            if (c.more > again.size()) {
                again.resize(c.more);
                d2h(again.data(), s.again, c.more * sizeof(MsdBucket));
                e = held.wait();
                if (e != cudaSuccess) return int(e);
            }
            for (const MsdBucket& b : again)
                work.push_back({b.start, b.start + b.size, int(b.id_off >> kIdBits), b.id_off & ((1u << kIdBits) - 1), false});
        }
    }
    if (own_span && c0.more) span(1);
    return int(cudaGetLastError());
}

struct SortOut {
    idx_t* sa;
    uint8_t* bwt;
    idx_t* kt;
    uint16_t* kx;
    int kx_bases;
    int kmer_k;
    bool kmer_spans;        // k-mers shorter than the buckets' prefix (or a chunk boundary's)
    bool kmer_done;
};

// The suffixes of at most S bases, if they are sorted apart: sorted and counted by bucket, and placed once
// the buckets' places are known.
struct ShortSuffixes {
    uint32_t* key;
    idx_t* val;
    size_t m;
    int sort(const MsdPlan& P, size_t nr, const MsdScratch& s, cudaStream_t st) {
        m = nr * size_t(P.S);
        if (!m) return 0;
        uint32_t *k0 = s.sk0, *k1 = s.sk1;
        idx_t *v0 = s.sv0, *v1 = s.sv1;
        k_short_keys<<<grid_for(m, 256), 256, 0, st>>>(s.pk, nr, P.dl.L, P.S, k0, v0);
        note_launch();
        const int rc = radix_sort_pairs<uint32_t, idx_t>(&k0, &v0, &k1, &v1, m, 0, P.S <= 3 ? 8 : 16, s.rtmp, s.rtmp_bytes, st, false);
        if (rc) return rc;
        key = k0;
        val = v0;
        cudaMemsetAsync(s.sfirst, 0xff, (size_t(1) << (P.d1 + P.d2)) * 8, st);
        k_short_runs<<<grid_for(m, 256), 256, 0, st>>>(s.pk, key, val, m, P.dl, P.d1 + P.d2, s.shorts, s.sfirst);
        note_launch();
        return 0;
    }
    void place(const MsdPlan& P, const MsdScratch& s, const SortOut& o, cudaStream_t st) const {
        if (!m) return;
        k_short_place<<<grid_for(m, 256), 256, 0, st>>>(s.pk, key, val, m, P.dl, P.d1 + P.d2, s.shorts, s.sfirst, s.lstart, o.sa, o.bwt,
                                                        o.kmer_k <= P.S ? o.kt : nullptr, o.kmer_k, o.kx, 2 * o.kx_bases);
        note_launch();
    }
};

// The listed buckets of the m suffixes from row `row0` on finished: at most `buckets` small ones, then the
// larger, their groups and what has to be split further (through `tmp`, m elements).
template <int W>
int msd_finish(const MsdPlan& P, const MsdScratch& s, const SortOut& o, const MsdLists& G, size_t row0, size_t m, size_t buckets,
               uint64_t* tmp, int sms, cudaStream_t st) {
    MsdLocal a{};
    a.plan = P;
    a.pk = s.pk;
    a.buf = s.b;
    a.G = G;
    a.sa = o.sa + row0;
    a.bwt = o.bwt ? o.bwt + row0 : nullptr;
    a.kt = o.kt;
    a.kx = o.kx ? o.kx + row0 : nullptr;
    a.kx_bits = 2 * o.kx_bases;
    a.kx_shift = P.key_shift + P.kbits - (2 * o.kmer_k - P.d1) - 2 * o.kx_bases;
    a.kmer_k = o.kmer_k;
    a.kmer_spans = o.kmer_spans;
    a.row0 = row0;
    a.more_bits = P.kbits & ~1;
    MsdKernels<W>::local(false, a, s, buckets, sms, st);
    MsdKernels<W>::local(true, a, s, m / kLocalSmall + 1, sms, st);
    MsdKernels<W>::groups(a, s, sms, st);
    MsdCounters c;
    cudaMemcpyAsync(&c, s.counters, sizeof c, cudaMemcpyDeviceToHost, st);
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return int(e);
    if (c.mid > s.cap_mid || c.big > s.cap_big) return int(cudaErrorUnknown);
    if (c.more || c.huge) {
        const int rc = more_splits<W>(c, a, s, tmp, sms, st);
        if (rc) return rc;
    }
    return int(cudaGetLastError());
}

// One chunk (or everything): the suffixes whose 6-base bucket lies in [c0, c1), m of them from row
// `row0` on; hist6 (host) holds a chunked sort's 6-base bucket counts.
template <int W>
int msd_pass(const MsdPlan& P, size_t nr, const MsdScratch& s, const SortOut& o, size_t row0, size_t m, uint32_t c0, uint32_t c1,
             const unsigned long long* hist6, size_t cap, bool* listed_more, cudaStream_t st) {
    const int sms = device_sms();
    const size_t bins1 = size_t(1) << P.d1;
    const int bits = P.d1 + P.d2;
    uint64_t* const ea = sizeof(idx_t) == 8 ? reinterpret_cast<uint64_t*>(o.sa + row0) : s.a;
    MsdLists G{s.small, s.large, s.more, s.mid, s.big, s.huge, s.cap_more, s.cap_mid, s.cap_big, s.cap_huge, s.counters};
    const size_t tiles = (P.n + kSplitTile - 1) / kSplitTile;
    const unsigned wide = unsigned(std::min<size_t>(tiles, size_t(sms) * 2));
    const size_t smem_text = MsdSmem::bytes(P.d1, true), smem_split = MsdSmem::bytes(std::max(P.d2, kMoreBits), false);
    const cudaError_t allowed = MsdKernels<W>::prepare();
    if (allowed != cudaSuccess) return int(allowed);

    cudaMemsetAsync(s.counters, 0, s.clear_bytes, st);
    if (hist6) {
        std::vector<unsigned long long> h(bins1, 0);
        for (uint32_t c = c0; c < c1; ++c) h[(c >> 3) >> (2 * kBucketBases - P.d1)] += hist6[c];
        cudaMemcpyAsync(s.hist, h.data(), bins1 * 8, cudaMemcpyHostToDevice, st);
        const cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return int(e);
    } else {
        k_msd_hist<<<unsigned(std::min<size_t>(tiles, size_t(sms) * 4)), kSplitThreads, 0, st>>>(s.pk, P, s.hist);
        note_launch();
    }
    ShortSuffixes sh{};
    if (const int rc = sh.sort(P, nr, s, st)) return rc;
    if (!P.d2) {
        k_msd_children<<<1, kScanThreads, 0, st>>>(s.hist, P.S ? s.shorts : nullptr, P.d1, 1, nullptr, s.lstart, s.cursor, 1, G);
        k_msd_text<uint64_t><<<wide, kSplitThreads, smem_text, st>>>(s.pk, P, s.cursor, s.b, c0, c1);
        const cudaError_t e = cudaGetLastError();           // the next kernels index by what these leave
        if (e != cudaSuccess) return int(e);
        note_launch();
        note_launch();
    } else {
        k_msd_children<<<1, kScanThreads, 0, st>>>(s.hist, nullptr, P.d1, 1, nullptr, s.start1, s.cursor1, 0, G);
        k_msd_text<uint64_t><<<wide, kSplitThreads, smem_text, st>>>(s.pk, P, s.cursor1, ea, c0, c1);
        const cudaError_t et = cudaGetLastError();          // the next kernels index by what these leave
        if (et != cudaSuccess) return int(et);
        k_msd_tiles<<<1, 1024, 0, st>>>(s.start1, s.cursor1, int(bins1), s.tile0);
        MsdRanges r{};
        r.start = s.start1;
        r.end = s.cursor1;
        r.tile0 = s.tile0;
        r.ushift = P.key_shift + P.kbits - P.d2;
        r.count = int(bins1);
        r.bits = P.d2;
        k_msd_count<<<unsigned(sms * 4), kSplitThreads, 0, st>>>(ea, r, s.cnt);
        k_msd_children<<<unsigned(bins1), kScanThreads, 0, st>>>(s.cnt, P.S ? s.shorts : nullptr, P.d2, 0, s.start1, s.lstart,
                                                                 s.cursor, 1, G);
        k_msd_split<<<unsigned(sms * 2), kSplitThreads, smem_split, st>>>(ea, r, s.cursor, s.b);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return int(e);
        for (int i = 0; i < 6; ++i) note_launch();
    }
    sh.place(P, s, o, st);
    std::vector<unsigned long long> h(cap ? bins1 : 0);
    if (cap) cudaMemcpyAsync(h.data(), s.hist, bins1 * 8, cudaMemcpyDeviceToHost, st);
    const int rc = msd_finish<W>(P, s, o, G, row0, m, size_t(1) << bits, ea, sms, st);
    if (rc) return rc;
    for (unsigned long long x : h)
        if (x > cap) *listed_more = true;           // (the caller looks at the 6-base buckets)
    return 0;
}

// A chunked sort of two passes: the first pass goes over the text once, into the suffix array itself (64-bit:
// its elements, 32-bit: positions, of which a chunk's elements are made when its turn comes); then runs
// of consecutive first-level buckets of at most `cap` suffixes are split and finished one after the other.
// A pass over the text for every chunk, as where a first-level bucket exceeds the chunk (*fits false,
// nothing written), costs chunks times n: 100 M suffixes in 40 chunks took 45.1 ms (radix passes of
// scattered positions 28.3), now 8.7; 1 G in 8 chunks 106 (91), now 46.
template <int W>
int msd_slices(const MsdPlan& P, size_t nr, const MsdScratch& s, const SortOut& o, size_t cap, bool* fits, cudaStream_t st) {
    const int sms = device_sms();
    const size_t bins1 = size_t(1) << P.d1;
    const MsdLists G{s.small, s.large, s.more, s.mid, s.big, s.huge, s.cap_more, s.cap_mid, s.cap_big, s.cap_huge, s.counters};
    const size_t tiles = (P.n + kSplitTile - 1) / kSplitTile;
    const cudaError_t allowed = MsdKernels<W>::prepare();
    if (allowed != cudaSuccess) return int(allowed);
    cudaMemsetAsync(s.counters, 0, s.clear_bytes, st);
    k_msd_hist<<<unsigned(std::min<size_t>(tiles, size_t(sms) * 4)), kSplitThreads, 0, st>>>(s.pk, P, s.hist);
    k_msd_children<<<1, kScanThreads, 0, st>>>(s.hist, nullptr, P.d1, 1, nullptr, s.start1, s.cursor1, 0, G);
    std::vector<unsigned long long> h(bins1);
    cudaMemcpyAsync(h.data(), s.hist, bins1 * 8, cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return int(e);
    *fits = *std::max_element(h.begin(), h.end()) <= cap;
    if (!*fits) return 0;
    ShortSuffixes sh{};
    if (const int rc = sh.sort(P, nr, s, st)) return rc;
    const unsigned wide = unsigned(std::min<size_t>(tiles, size_t(sms) * 2));
    k_msd_text<idx_t><<<wide, kSplitThreads, MsdSmem::bytes(P.d1, true), st>>>(s.pk, P, s.cursor1, o.sa, 0, uint32_t(kBuckets));
    e = cudaGetLastError();                                 // the next kernels index by what these leave
    if (e != cudaSuccess) return int(e);
    for (int i = 0; i < 3; ++i) note_launch();
    size_t row = 0;
    for (size_t lo = 0, hi; lo < bins1; lo = hi) {
        size_t m = 0;
        for (hi = lo; hi < bins1 && m + h[hi] <= cap; ++hi) m += size_t(h[hi]);
        if (!m) continue;
        cudaMemsetAsync(s.counters, 0, sizeof(MsdCounters), st);
        const uint64_t* in = reinterpret_cast<const uint64_t*>(o.sa);
        MsdRanges r{};
        r.start = s.start1 + lo;
        r.end = s.cursor1 + lo;
        r.tile0 = s.tile0;
        r.ushift = P.key_shift + P.kbits - P.d2;
        r.count = int(hi - lo);
        r.bits = P.d2;
        k_msd_tiles<<<1, 1024, 0, st>>>(r.start, r.end, r.count, s.tile0);
        if (sizeof(idx_t) == 4) {
            r.base = row;
            k_msd_gather<<<unsigned(sms * 4), kSplitThreads, 0, st>>>(s.pk, P, o.sa, r, s.a);
            note_launch();
            in = s.a;
        }
        k_msd_count<<<unsigned(sms * 4), kSplitThreads, 0, st>>>(in, r, s.cnt + (lo << P.d2));
        k_msd_children<<<unsigned(hi - lo), kScanThreads, 0, st>>>(s.cnt, P.S ? s.shorts : nullptr, P.d2, 0, s.start1, s.lstart, s.cursor, 1, G,
                                                                  unsigned(lo), row);
        k_msd_split<<<unsigned(sms * 2), kSplitThreads, MsdSmem::bytes(P.d2, false), st>>>(in, r, s.cursor + (lo << P.d2), s.b);
        e = cudaGetLastError();
        if (e != cudaSuccess) return int(e);
        for (int i = 0; i < 4; ++i) note_launch();
        uint64_t* const tmp = sizeof(idx_t) == 8 ? reinterpret_cast<uint64_t*>(o.sa + row) : s.a;
        const int rc = msd_finish<W>(P, s, o, G, row, m, (hi - lo) << P.d2, tmp, sms, st);
        if (rc) return rc;
        row += m;
    }
    sh.place(P, s, o, st);
    return int(cudaGetLastError());
}

}  // namespace

size_t suffix_sort_tmp_bytes(size_t n, size_t num_reads, int L, size_t cap) {
    return n ? sort_shape(n, num_reads, L, cap).bytes : 0;
}

// Prefix doubling on 29-base keys (reads longer than the networks' words).
static int sort_doubling(size_t n, int L, idx_t* sa, const uint64_t* pk, void* tmp, cudaStream_t st) {
    char* p = static_cast<char*>(tmp);
    uint64_t* ka = reinterpret_cast<uint64_t*>(p); p += al(n * sizeof(uint64_t));
    uint64_t* kb = reinterpret_cast<uint64_t*>(p); p += al(n * sizeof(uint64_t));
    idx_t* va = sa;
    idx_t* vb = reinterpret_cast<idx_t*>(p); p += al(n * sizeof(idx_t));
    uint32_t* rank = reinterpret_cast<uint32_t*>(p); p += al(n * sizeof(uint32_t));
    p += al((n / 32 + 4) * sizeof(uint64_t));           // packed text, when the caller keeps none
    void* rtmp = p; p += al(radix_tmp_bytes(n));
    const size_t tiles = (n + HT_TILE - 1) / HT_TILE;
    unsigned long long* tmax = reinterpret_cast<unsigned long long*>(p);
    unsigned long long* tcnt = tmax + tiles + 1;
    unsigned long long* groups = tcnt + tiles + 1;
    { k_init_keys<<<grid_for(n, 256), 256, 0, st>>>(pk, n, idx_t(L), ka, va); note_launch(); }
    int rc = radix_sort_pairs<uint64_t, idx_t>(&ka, &va, &kb, &vb, n, 0, 64, rtmp, radix_tmp_bytes(n), st, true);
    if (rc) return rc;
    for (size_t h = kWide;; h *= 2) {
        { k_head_tiles<<<unsigned(tiles), HT_THREADS, 0, st>>>(ka, n, tmax, tcnt); note_launch(); }
        { k_head_carry<<<1, 1024, 0, st>>>(tmax, tcnt, tiles, groups); note_launch(); }
        { k_head_apply<idx_t><<<unsigned(tiles), HT_THREADS, 0, st>>>(ka, kb, va, n, tmax, rank); note_launch(); }
        std::swap(ka, kb);
        unsigned long long g = 0;
        cudaMemcpyAsync(&g, groups, sizeof g, cudaMemcpyDeviceToHost, st);
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return int(e);
        if (g == n || h >= size_t(L)) break;
        { k_second_keys<idx_t><<<grid_for(n, 256), 256, 0, st>>>(ka, va, n, idx_t(L), h, rank); note_launch(); }
        int bits = 1;
        while ((size_t(1) << bits) <= n + 1) ++bits;
        rc = radix_sort_pairs<uint64_t, idx_t>(&ka, &va, &kb, &vb, n, 0, 32 + bits, rtmp, radix_tmp_bytes(n), st, true);
        if (rc) return rc;
    }
    if (va != sa) { k_copy_vals<idx_t><<<grid_for(n, 256), 256, 0, st>>>(va, n, sa); note_launch(); }
    return int(cudaGetLastError());
}

// A chunked sort's bucket histogram: 6-base buckets counted in shared memory (kBuckets 32-bit
// counters, one CTA per SM) and added to the global histogram once per CTA.
constexpr int kHistThreads = 1024;
__global__ void __launch_bounds__(kHistThreads) k_bucket_hist(const uint64_t* __restrict__ pk, size_t n, DivL dl,
                                                              unsigned long long* __restrict__ hist) {
    extern __shared__ unsigned s_hist[];
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    const size_t stride = size_t(gridDim.x) * kHistThreads * 16;
    for (size_t p0 = (size_t(blockIdx.x) * kHistThreads + threadIdx.x) * 16; p0 < n; p0 += stride)
        for_positions(pk, p0, n, dl, [&](int, size_t, uint64_t x, int m, int, bool) { atomicAdd(&s_hist[bucket6(x, m)], 1u); });
    __syncthreads();
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x)
        if (s_hist[i]) atomicAdd(&hist[i], (unsigned long long)s_hist[i]);
}

static int bucket_hist(const uint64_t* pk, size_t n, const DivL& dl, unsigned long long* dev, std::vector<unsigned long long>& h,
                       cudaStream_t st) {
    constexpr size_t hsm = size_t(kBuckets) * sizeof(unsigned);
    const cudaError_t allowed = allow_smem<hsm>(k_bucket_hist);
    if (allowed != cudaSuccess) return int(allowed);
    cudaMemsetAsync(dev, 0, size_t(kBuckets) * 8, st);
    { k_bucket_hist<<<unsigned(device_sms()), kHistThreads, hsm, st>>>(pk, n, dl, dev); note_launch(); }
    h.resize(kBuckets);
    cudaMemcpyAsync(h.data(), dev, size_t(kBuckets) * 8, cudaMemcpyDeviceToHost, st);
    return int(cudaStreamSynchronize(st));
}

template <int W>
static int sort_msd(const SortShape& sh, size_t nr, const MsdScratch& s, SortOut& o, size_t cap, cudaStream_t st) {
    const MsdPlan& P = sh.plan;
    const size_t n = P.n;
    // k-mers entered as the buckets finish: of up to `head` bases; where they span buckets or short
    // suffixes have them too, by minimum and maximum
    if (o.kt && o.kmer_k > P.head) o.kt = nullptr;
    o.kx_bases = o.kt && o.kx && 2 * o.kmer_k >= P.d1 ? std::min(7, P.head - o.kmer_k) : 0;
    if (!o.kx_bases) o.kx = nullptr;
    const bool spans = o.kmer_spans = o.kmer_k <= P.S || 2 * o.kmer_k < std::max(P.d1 + P.d2, sh.chunked ? 2 * kBucketBases : 0);
    const size_t nk = size_t(1) << (2 * o.kmer_k);
    if (o.kt && spans) { k_kmer_span<<<grid_for(nk, 256), 256, 0, st>>>(o.kt, nk, 0, nullptr, 0); note_launch(); }
    if (o.kt && !spans) {
        const cudaError_t e = kmer_table_clear(o.kmer_k, o.kt, st);
        if (e != cudaSuccess) return int(e);
    }
    bool more = false;
    std::vector<unsigned long long> h6;
    if (!sh.chunked) {
        const int rc = msd_pass<W>(P, nr, s, o, 0, n, 0, uint32_t(kBuckets), nullptr, cap, &more, st);
        if (rc) return rc;
        if (more) {       // a first-level bucket above the chunk size: is a 6-base one?
            const int rh = bucket_hist(s.pk, n, P.dl, s.hist6, h6, st);
            if (rh) return rh;
            for (unsigned long long x : h6)
                if (x > cap) return int(cudaErrorNotSupported);
        }
    } else {
        bool fits = false;
        if (P.d2) {
            const int rc = msd_slices<W>(P, nr, s, o, cap, &fits, st);
            if (rc) return rc;
        }
        MsdPlan Q = P;              // by a pass over the text a chunk: short suffixes like all others
        Q.S = 0;
        const int rh = fits ? 0 : bucket_hist(s.pk, n, P.dl, s.hist6, h6, st);
        if (rh) return rh;
        for (unsigned long long x : h6)
            if (x > cap) return int(cudaErrorNotSupported);              // one bucket larger than a chunk
        // chunks: runs of consecutive buckets that fit the capacity, each a slice of the suffix array
        size_t row = 0;
        for (uint32_t lo = fits ? uint32_t(kBuckets) : 0; lo < uint32_t(kBuckets);) {
            uint32_t hi = lo;
            size_t m = 0;
            while (hi < uint32_t(kBuckets) && m + h6[hi] <= cap) m += h6[hi++];
            if (m) {
                const int rc = msd_pass<W>(Q, nr, s, o, row, m, lo, hi, h6.data(), 0, &more, st);
                if (rc) return rc;
            }
            row += m;
            lo = hi;
        }
    }
    if (o.kt && spans) { k_kmer_span<<<grid_for(nk, 256), 256, 0, st>>>(o.kt, nk, 1, nullptr, 0); note_launch(); }
    o.kmer_done = o.kt != nullptr;
    return int(cudaGetLastError());
}

int suffix_sort(const uint8_t* reads, idx_t num_reads, int L, int dir, idx_t* sa, size_t cap, void* tmp,
                size_t tmp_bytes, cudaStream_t st, const uint8_t** bwt_out, uint64_t* pk_out, idx_t* kt, int kmer_k, bool* kmer_done,
                uint16_t* kx, int* kx_bases) {
    if (bwt_out) *bwt_out = nullptr;
    if (kmer_done) *kmer_done = false;
    if (kx_bases) *kx_bases = 0;
    const size_t n = size_t(num_reads) * size_t(L);
    if (n == 0) return 0;
    if (cap >= n) cap = 0;
    if (cap == 1) return int(cudaErrorInvalidValue);
    const SortShape sh = sort_shape(n, num_reads, L, cap);
    if (tmp_bytes < sh.bytes) return int(cudaErrorInvalidValue);
    if (cap && L > kChunkMaxLen) return int(cudaErrorNotSupported);
    if (sh.doubling && n >= (size_t(1) << 31)) return int(cudaErrorNotSupported);      // 32-bit ranks
    MsdScratch s{};
    if (!sh.doubling) s = msd_layout(tmp, sh.plan, sh.m, num_reads);
    uint64_t* pk = pk_out;
    if (!pk) {
        if (!sh.doubling) pk = s.pk;
        else pk = reinterpret_cast<uint64_t*>(static_cast<char*>(tmp) + 2 * al(n * sizeof(uint64_t)) + al(n * sizeof(idx_t)) +
                                              al(n * sizeof(uint32_t)));
    }
    const size_t nwords = n / 32 + 4;
    { k_pack_text<<<grid_for(nwords, 256), 256, 0, st>>>(reads, n, make_divl(uint32_t(L)), dir, nwords, pk); note_launch(); }
    if (sh.doubling) return sort_doubling(n, L, sa, pk, tmp, st);
    s.pk = pk;
    SortOut o{sa, bwt_out ? s.bwt : nullptr, kt, kx, 0, kmer_k, false, false};
    int rc = 0;
    switch (plan_words(sh.plan)) {
        case 1: rc = sort_msd<1>(sh, num_reads, s, o, cap, st); break;
        case 2: rc = sort_msd<2>(sh, num_reads, s, o, cap, st); break;
        case 3: rc = sort_msd<3>(sh, num_reads, s, o, cap, st); break;
        case 4: rc = sort_msd<4>(sh, num_reads, s, o, cap, st); break;
        case 5: rc = sort_msd<5>(sh, num_reads, s, o, cap, st); break;
        case 6: rc = sort_msd<6>(sh, num_reads, s, o, cap, st); break;
        case 7: rc = sort_msd<7>(sh, num_reads, s, o, cap, st); break;
        case 8: rc = sort_msd<8>(sh, num_reads, s, o, cap, st); break;
        default: rc = sort_msd<9>(sh, num_reads, s, o, cap, st); break;
    }
    if (rc) return rc;
    if (bwt_out) *bwt_out = s.bwt;
    if (kmer_done) *kmer_done = o.kmer_done;
    if (kx_bases) *kx_bases = o.kx_bases;
    return 0;
}

}  // namespace pq
