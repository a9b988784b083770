// pq_search.cu — per-read overlap search with transitive reduction on the GPU.
//
// Replaces the body of construct_string_graph's per-read loop (src/string_graph.c:800-830):
//   find_intervals   (src/string_graph.c:163-383)  four bidirectional backward searches
//   extract_bw_edges (src/string_graph.c:560-731)  DFS irreducible-edge extraction, B side
//   extract_fw_edges (src/string_graph.c:387-556)  the same for the F side
// with the rank primitives OCCx/search_1/search_2/search_3 (src/string_graph.c:11-159) on the
// one-sector occ blocks of pq_common.cuh.
//
// Tiers, each of which lists the reads it cannot hold for a later one, so that every read completes
// with the reference's result: the lean tier (a warp takes up to 32 reads' rows of the suffix array and
// reduces their candidates by sorted continuations), the block tier (a CTA a read, the same by sorting in
// shared or global memory), the fast and the heavy tier (the reference's walk and DFS, a read a lane,
// intervals spread over the warp), and the wide tier, one thread a read: candidate intervals of every open
// level in an array laid out as the reference's I_fw/I_bw (a level's children directly after it), one frame per
// level for the extension base that comes next, and the reference's own bounds ((2L)^2 candidates, 65535
// edges per side).
#include "pq_index.cuh"
#include "pq_learned.cuh"

#include <algorithm>

namespace pq {

// One candidate interval (interval_t, src/string_graph.h:47-54).  Its remaining size is always
// uu - ll + 1 here: zero-$ level-0 entries are not stored (see side_candidates) and no counter is
// decremented, so the field is not kept.
struct Cand {
    idx_t ll, uu;
    uint16_t len;
    uint8_t type;
};
struct Frame {
    uint32_t pos;       // first candidate of this level
    uint32_t free;      // first stack slot this level may use for its extension sets
    uint32_t cbase;     // first slot of the four extension sets (stored back to back, A..T)
    int32_t trans;      // sum of this level's interval sizes (path_t.trans of its edges)
    uint16_t size;
    uint16_t maxlen;
    uint16_t csz[4];    // non-empty extensions by A, C, G, T
    uint8_t next_a;
};
struct EdgeRec {
    idx_t dest;
    int32_t trans;
    uint16_t len;
    uint8_t type;
};

// Per-thread counters of a search: rank probes (one occurrence block each, the unit of the
// reference's OCCx/search_* calls) and the 32-byte sectors of every global load of index data the
// method issues -- occurrence blocks, k-mer table entries and next bases, suffix-array entries,
// packed-text words, reads_index entries and read bytes.  Tables that stay resident in L2 (the
// superblock counts, learned models) and the search's own scratch are not counted.  `+= n` is n
// rank probes, one sector each (an occurrence block is one aligned sector).
struct Tally {
    uint32_t probes{0}, sectors{0};
    __device__ __forceinline__ Tally& operator+=(uint32_t n) {
        probes += n;
        sectors += n;
        return *this;
    }
    __device__ __forceinline__ void add(uint32_t p, uint32_t s) {
        probes += p;
        sectors += s;
    }
};

// bases from text position p to the end of its read, and the read of position p (DivL: no divide)
__device__ __forceinline__ int suffix_len(idx_t p, const DivL& dl) {
    return int(dl.L - uint32_t(uint64_t(p) - div_l(uint64_t(p), dl) * dl.L));
}
__device__ __forceinline__ idx_t read_of(idx_t p, const DivL& dl) { return idx_t(div_l(uint64_t(p), dl)); }

// 32-byte sectors spanned by `bytes` bytes at p
__device__ __forceinline__ uint32_t sectors_of(const void* p, size_t bytes) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    return uint32_t(((a + bytes - 1) >> 5) - (a >> 5) + 1);
}

// ------------------------------------------------------------------------------ rank primitives

__device__ __forceinline__ void ld_block(const OccBlock* p, uint64_t& lo, uint64_t& hi, uint64_t& dol,
                                         uint32_t& c01, uint32_t& c23) {
    const uint4* q = reinterpret_cast<const uint4*>(p);
    uint4 a = __ldg(q);
    uint4 b = __ldg(q + 1);
    lo = uint64_t(a.x) | (uint64_t(a.y) << 32);
    hi = uint64_t(a.z) | (uint64_t(a.w) << 32);
    dol = uint64_t(b.x) | (uint64_t(b.y) << 32);
    c01 = b.z;
    c23 = b.w;
}

__device__ __forceinline__ uint64_t below(idx_t pos) {
    return (uint64_t(1) << (pos & 63)) - 1;   // rows [64*(pos/64), pos) of the block
}

// match mask of base c (1..4) among non-$ rows
__device__ __forceinline__ uint64_t match(uint64_t lo, uint64_t hi, uint64_t dol, int c) {
    uint64_t code = uint64_t(c - 1);
    uint64_t mlo = lo ^ ((code & 1) - 1);
    uint64_t mhi = hi ^ ((code >> 1) - 1);
    return mlo & mhi & ~dol;
}

__device__ __forceinline__ uint32_t rel_cnt(uint32_t c01, uint32_t c23, int c) {
    uint32_t w = (c <= 2) ? c01 : c23;
    return ((c & 1) ? w : (w >> 16)) & 0xffff;
}

// ranks of all four bases in BWT[0, pos)
__device__ __forceinline__ void rank_all(const FmView& f, idx_t pos, idx_t r[4]) {
    uint64_t lo, hi, dol;
    uint32_t c01, c23;
    ld_block(f.blk + (pos >> kBlockShift), lo, hi, dol, c01, c23);
    const idx_t* s4 = f.sb + size_t(pos >> kSuperShift) * 4;
    idx_t s0, s1, s2, s3;
#ifdef PQ_IDX64
    ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2*>(s4));
    ulonglong2 b = __ldg(reinterpret_cast<const ulonglong2*>(s4) + 1);
    s0 = a.x; s1 = a.y; s2 = b.x; s3 = b.y;
#else
    uint4 a = __ldg(reinterpret_cast<const uint4*>(s4));
    s0 = a.x; s1 = a.y; s2 = a.z; s3 = a.w;
#endif
    uint64_t m = below(pos) & ~dol;
    r[0] = s0 + (c01 & 0xffff) + idx_t(__popcll(~hi & ~lo & m));
    r[1] = s1 + (c01 >> 16) + idx_t(__popcll(~hi & lo & m));
    r[2] = s2 + (c23 & 0xffff) + idx_t(__popcll(hi & ~lo & m));
    r[3] = s3 + (c23 >> 16) + idx_t(__popcll(hi & lo & m));
}

// # of `$` rows in BWT[0, pos) (= the reference's OCC(0, pos))
__device__ __forceinline__ idx_t rank_dollar(const FmView& f, idx_t pos) {
    idx_t r[4];
    rank_all(f, pos, r);
    return pos - (r[0] + r[1] + r[2] + r[3]);
}

// ------------------------------------------------------------------------------ per-read search

struct ReadView {
    const uint32_t* w;   // packed 2-bit codes (A=0..T=3), 16 per word, word i at w[i*stride]
    int stride;
    __device__ __forceinline__ int at(int i) const {   // code 1..4 of read position i
        return int((w[(i >> 4) * stride] >> ((i & 15) * 2)) & 3) + 1;
    }
};

__device__ __forceinline__ int complement(int c) { return 5 - c; }

// pattern base at depth j (1-based) of each search kind (see oracle candidate_search)
__device__ __forceinline__ int pattern_at(const ReadView& rd, int L, int kind, int j) {
    switch (kind) {
        case PQ_FB: return rd.at(L - j);
        case PQ_FF: return complement(rd.at(L - j));
        case PQ_BF: return rd.at(j - 1);
        default: return complement(rd.at(j - 1));
    }
}

// first and last row of a k-mer (last < first when it is absent)
__device__ __forceinline__ void kmer_rows(const FmView& f, uint32_t code, idx_t& first, idx_t& last) {
#ifdef PQ_IDX64
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(f.kt) + code);
#else
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(f.kt) + code);
#endif
    first = v.x;
    last = v.y;
}

// exact SA interval of pattern pat(hi) pat(hi-1) ... pat(lo) (text order) from the k-mer table
__device__ __forceinline__ void kmer_seed(const FmView& f, const ReadView& rd, int L, int kind, int first,
                                          int last, int step, idx_t& l, idx_t& u, Tally& probes) {
    uint32_t code = 0;
    for (int j = first;; j += step) {
        code = (code << 2) | uint32_t(pattern_at(rd, L, kind, j) - 1);
        if (j == last) break;
    }
    kmer_rows(f, code, l, u);
    probes.add(1, 1);
}

struct ReadResult {
    int status;
    int nB, nF;
    int32_t olpB, olpF;
    int ne;
};

__device__ __forceinline__ idx_t pick4(const idx_t r[4], int c) {   // r[c - 1] without local memory
    return c == 1 ? r[0] : (c == 2 ? r[1] : (c == 3 ? r[2] : r[3]));
}

// search_2 from ranks already loaded at vl = l and vu = u + 1 (the same two blocks also give the
// `$` count of search_3, so one pair of loads serves both).
__device__ __forceinline__ void step_from_ranks(const FmView& f, int c, idx_t vl, idx_t vu, const idx_t rl[4],
                                                const idx_t ru[4], idx_t& l, idx_t& u, idx_t& ll, idx_t& uu) {
    idx_t gel = 0, geu = 0;
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (k + 1 >= c) { gel += rl[k]; geu += ru[k]; }
    }
    ll = ll + ((vu - geu) - (vl - gel));
    const idx_t ol = pick4(rl, c), ou = pick4(ru, c);
    const idx_t base = f.Cf[c];
    l = base + ol;
    u = base + ou - 1;
    uu = ll + ou - ol - 1;
}

__device__ __forceinline__ bool live(int kind, idx_t l, idx_t u) {
    return (kind == PQ_FB || kind == PQ_BF) ? (l < u) : (l <= u);   // src/string_graph.c:207 vs :251
}
__device__ __forceinline__ int walked_index(int kind) { return (kind == PQ_FB || kind == PQ_BB) ? 0 : 1; }

__device__ __forceinline__ uint32_t pack_meta(int len, int type) { return uint32_t(len) | (uint32_t(type) << 16); }
__device__ __forceinline__ int meta_len(uint32_t m) { return int(m & 0xffff); }
__device__ __forceinline__ int meta_type(uint32_t m) { return int(m >> 16); }

// ---------------------------------------------------------------- candidates by interval scan
//
// A candidate of kind `kind` at depth d (t <= d < L) is a read r' whose first d bases, in the
// walked index's text, equal P_d = pat(d) .. pat(1).  Its last t bases there are P_t, so r'
// appears in the depth-t interval I_t of the walked index as the row of its suffix at offset
// o = d - t; conversely a row (r', o) of I_t with o < L - t is a candidate at depth t + o exactly
// when r'[0, o) = pat(t + o) .. pat(t + 1).  So instead of walking from depth t to L one base at a
// time (the reference's search_2/search_3 loop, src/string_graph.c:226-237), the rows of I_t are
// read once: one suffix-array entry and one text comparison each, all independent loads.
//
// Chains are alive at depth d whenever a candidate exists there (a strict kind also holds the
// read's own suffix, a second row), so the depths reported are the reference's.  I_t itself is not
// needed row for row: any run of rows that holds it serves, since every row is checked against the
// whole pattern P_d.  That run is the rows of P_t's first k bases (k-mer table) that go on with its
// next kx_bases bases (FmView::kx); a run of more than kScanDirect rows, or the window of the
// learned index, is narrowed to I_t by binary search over the suffix array.

constexpr int kScanWords = 2;       // bases of P_t searched by bisection: the first 64 at most
constexpr int kScanMax = 256;       // larger depth-t intervals walk instead
constexpr int kScanDirect = 48;     // rows checked without narrowing them to I_t first,
constexpr int kScanBare = 8;        // where no next bases have narrowed them: a row of a k-mer may be of I_t by
                                    // chance only (0.4 M reads of 76 random bases, 20 % GC: 0.41 ms with 48, 0.23; 30x
                                    // of a genome, 100 bases, 0.38 and 0.33).  Not where a warp has fewer than 32 reads,
                                    // which wait for the bisection (20 thousand reads: 0.10 with 48, 0.12), nor for reads
                                    // of up to 64 bases, whose k-mers have few rows (61 bases at 20x: 0.28 and 0.30)

// 32 bases of packed text starting at base p (first base in the top bits)
__device__ __forceinline__ uint64_t text_window(const uint64_t* __restrict__ pk, size_t p) {
    const size_t w = p >> 5;
    const int s = int(p & 31) * 2;
    const uint64_t a = __ldg(pk + w), b = __ldg(pk + w + 1);
    return s ? ((a << s) | (b >> (64 - s))) : a;
}

__device__ __forceinline__ uint64_t top_mask(int nbases) {      // 1 <= nbases <= 32
    return nbases >= 32 ? ~uint64_t(0) : ~(~uint64_t(0) >> (2 * nbases));
}

// P = pat(t) .. pat(1) of `kind` in the walked index's text order, its first 64 bases packed (the
// bases past t are whatever follows; every comparison masks them).  P is the read's own text in
// the walked index at self * L + L - t for a strict kind, and the complement of the other index's
// text there for FF and BB.
__device__ __forceinline__ void pattern_words(const FmView* fm, int L, int t, int kind, idx_t self,
                                              uint64_t (&P)[kScanWords], Tally& probes) {
    const bool strict = kind == PQ_FB || kind == PQ_BF;
    const uint64_t* pk = fm[strict ? walked_index(kind) : 1 - walked_index(kind)].pk;
    const size_t pos = size_t(self) * L + size_t(L - t);
    const uint64_t flip = strict ? 0 : ~uint64_t(0);
    #pragma unroll
    for (int w = 0; w < kScanWords; ++w) P[w] = text_window(pk, pos + 32 * w) ^ flip;
    probes.add(0, sectors_of(pk + (pos >> 5), 8 * (kScanWords + 1)));
}

// -1 / 0 / +1: the suffix at text position p (m bases to end-of-read) is below / starts with /
// above P (t bases)
__device__ __forceinline__ int cmp_row(const uint64_t* __restrict__ pk, idx_t p, int m,
                                       const uint64_t (&P)[kScanWords], int t) {
    const int nb = m < t ? m : t;
    const size_t w0 = size_t(p) >> 5;
    const int s = int(p & 31) * 2;
    const uint64_t a = __ldg(pk + w0), b = __ldg(pk + w0 + 1), c = __ldg(pk + w0 + 2);
    const uint64_t x0 = s ? ((a << s) | (b >> (64 - s))) : a;
    const uint64_t x1 = s ? ((b << s) | (c >> (64 - s))) : b;
    const uint64_t k0 = top_mask(nb);
    if ((x0 & k0) != (P[0] & k0)) return (x0 & k0) < (P[0] & k0) ? -1 : 1;
    if (nb > 32) {
        const uint64_t k1 = top_mask(nb - 32);
        if ((x1 & k1) != (P[1] & k1)) return (x1 & k1) < (P[1] & k1) ? -1 : 1;
    }
    return m < t ? -1 : 0;
}

// sectors cmp_row loads for a suffix at text position p
__device__ __forceinline__ uint32_t cmp_sectors(const uint64_t* pk, idx_t p) {
    return sectors_of(pk + (size_t(p) >> 5), 24);
}

// Rows [first, end) of each chain's index that start with its pattern, searched within
// [lo, hi): lower and upper bounds of both chains advance together (four independent searches).
__device__ __forceinline__ void sa_bounds2(const FmView* f0, const FmView* f1, const DivL& dl,
                                           const uint64_t (&P0)[kScanWords],
                                           const uint64_t (&P1)[kScanWords], int t, const idx_t (&lo)[2],
                                           const idx_t (&hi)[2], idx_t (&first)[2], idx_t (&end)[2],
                                           Tally& probes) {
    idx_t a0[2] = {lo[0], lo[1]}, a1[2] = {hi[0], hi[1]}, b0[2] = {lo[0], lo[1]}, b1[2] = {hi[0], hi[1]};
    const FmView* fq[2] = {f0, f1};
    while (a0[0] < a1[0] || b0[0] < b1[0] || a0[1] < a1[1] || b0[1] < b1[1]) {
        idx_t pa[2], pb[2];
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            pa[q] = a0[q] < a1[q] ? __ldg(fq[q]->sa + (a0[q] + (a1[q] - a0[q]) / 2)) : 0;
            pb[q] = b0[q] < b1[q] ? __ldg(fq[q]->sa + (b0[q] + (b1[q] - b0[q]) / 2)) : 0;
        }
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint64_t (&P)[kScanWords] = q ? P1 : P0;
            if (a0[q] < a1[q]) {
                const idx_t ma = a0[q] + (a1[q] - a0[q]) / 2;
                const int c = cmp_row(fq[q]->pk, pa[q], suffix_len(pa[q], dl), P, t);
                if (c < 0) a0[q] = ma + 1;
                else a1[q] = ma;
                probes.add(2, 1 + cmp_sectors(fq[q]->pk, pa[q]));
            }
            if (b0[q] < b1[q]) {
                const idx_t mb = b0[q] + (b1[q] - b0[q]) / 2;
                const int c = cmp_row(fq[q]->pk, pb[q], suffix_len(pb[q], dl), P, t);
                if (c <= 0) b0[q] = mb + 1;
                else b1[q] = mb;
                probes.add(2, 1 + cmp_sectors(fq[q]->pk, pb[q]));
            }
        }
    }
    first[0] = a0[0]; first[1] = a0[1];
    end[0] = b0[0]; end[1] = b0[1];
}

// 32-byte sectors of packed text that hold the bases [p, p + m), m > 0 (the text starts on a sector)
__device__ __forceinline__ uint32_t base_sectors(size_t p, int m) { return uint32_t(((p + size_t(m) - 1) >> 7) - (p >> 7)) + 1u; }

// 32 bases from base offset s (0..31) of the words a, b (first base highest) as two 32-bit halves
__device__ __forceinline__ void shift_bases(uint64_t a, uint64_t b, int s, uint32_t& hi, uint32_t& lo) {
    const uint32_t r0 = uint32_t(a >> 32), r1 = uint32_t(a), r2 = uint32_t(b >> 32), r3 = uint32_t(b);
    const bool odd = s >= 16;
    const uint32_t h0 = odd ? r1 : r0, h1 = odd ? r2 : r1, h2 = odd ? r3 : r2;
    hi = __funnelshift_l(h1, h0, 2 * s);
    lo = __funnelshift_l(h2, h1, 2 * s);
}
// the bits of half h (0: the higher) of 32 bases that lie within the first `left` of them
__device__ __forceinline__ uint32_t half_mask(int left, int h) {
    uint32_t past;
    asm("shr.u32 %0, %1, %2;" : "=r"(past) : "r"(0xffffffffu), "r"(uint32_t(max(2 * left - 32 * h, 0))));   // 0 from 32 on
    return ~past;
}

// The d bases of the walked index's text at ra equal those of the pattern source at rs (their
// complement for cmpl), 32 at a time.  The pattern P_d of a strict kind is the read's own text in the
// walked index at self * L + L - d; of FF and BB it is the complement of the other index's text
// there.  Most rows compared do match, so nothing waits for the first difference: the warp runs to
// its longest d, each word loaded two steps ahead (no word past the one after the last base's: the
// text is padded by more).
__device__ __forceinline__ bool text_matches(const uint64_t* __restrict__ pka, size_t ra,
                                             const uint64_t* __restrict__ pks, size_t rs, int d, bool cmpl, unsigned lanes) {
    const uint64_t *wa = pka + (ra >> 5), *wb = pks + (rs >> 5);
    const int sa = int(ra & 31), sb = int(rs & 31), words = (d + 31) >> 5;
    const int most = int(__reduce_max_sync(lanes, unsigned(words)));
    const uint32_t flip = cmpl ? ~0u : 0u;
    uint64_t a0 = __ldg(wa), b0 = __ldg(wb), a1 = __ldg(wa + 1), b1 = __ldg(wb + 1);
    uint32_t x = 0;
    #pragma unroll 1
    for (int i = 0; i < most; ++i) {
        const int next = i + 2 < words ? i + 2 : words;
        const uint64_t a2 = __ldg(wa + next), b2 = __ldg(wb + next);
        const int left = d - 32 * i;
        uint32_t ah, al, bh, bl;
        shift_bases(a0, a1, sa, ah, al);
        shift_bases(b0, b1, sb, bh, bl);
        x |= ((ah ^ bh ^ flip) & half_mask(left, 0)) | ((al ^ bl ^ flip) & half_mask(left, 1));
        a0 = a1;
        b0 = b1;
        a1 = a2;
        b1 = b2;
    }
    return !x;
}

// Slots of the level-0 candidates of the two chains of one side: q * M + i.
struct SlotsFast {     // fast tier: the warp's global scratch, the lanes' slots interleaved
    idx_t* ll;
    idx_t* uu;
    uint32_t* meta;
    size_t base;
    int M;
    __device__ __forceinline__ void set(int q, int i, idx_t a, idx_t b, uint32_t m) const {
        const size_t p = base + (size_t(q) * M + i) * 32;
        ll[p] = a;
        uu[p] = b;
        meta[p] = m;
    }
};
struct SlotsStack {    // wide tier: the slot's candidate stack
    Cand* stk;
    int M;
    __device__ __forceinline__ void set(int q, int i, idx_t a, idx_t b, uint32_t m) const {
        Cand& c = stk[q * M + i];
        c.ll = a;
        c.uu = b;
        c.len = uint16_t(meta_len(m));
        c.type = uint8_t(meta_type(m));
    }
};

// find_intervals for one side: kinds k0 then k1 (B-F and B-B, or F-B and F-F), searched in
// lockstep so that each thread keeps two independent chains of loads in flight.
//
// The reference walks index A from its seed to depth t with search_1, then rebuilds the other
// index's interval of the reversed pattern from depth 1 with another t-1 search_1 steps, and
// only then continues with synchronised search_2 steps.  Here both intervals start from exact
// k-mer seeds (one per index) and every step is a synchronised step, so the other interval is
// known at every depth and the rebuild disappears; SA intervals are unique per string, so the
// intervals at depth t -- and everything after -- are the reference's.  The i-th stored candidate
// of kind k0 (q = 0) or k1 (q = 1) goes to slot (q, i); n[q] counts them.
template <class Slots>
__device__ __forceinline__ void chain_pair(const SearchArgs& A, const FmView* fm, const ReadView& rd, int k0, int k1,
                                           int (&n)[2], int32_t& olp, Tally& probes, const Slots& slots) {
    const int L = A.L, t = A.t, k = A.seed_k;
    n[0] = n[1] = 0;
    idx_t l[2], u[2], ll[2], uu[2];
    bool alive[2];
    #pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int kind = q ? k1 : k0;
        const int ia = walked_index(kind);
        kmer_seed(fm[ia], rd, L, kind, k, 1, -1, l[q], u[q], probes);       // pat(k) .. pat(1)
        kmer_seed(fm[1 - ia], rd, L, kind, 1, k, 1, ll[q], uu[q], probes);  // pat(1) .. pat(k)
        alive[q] = live(kind, l[q], u[q]);
    }
    int d = k;
    while (d < t && (alive[0] || alive[1])) {
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!alive[q]) continue;
            const int kind = q ? k1 : k0;
            const FmView& f = fm[walked_index(kind)];
            const idx_t vl = l[q], vu = u[q] + 1;
            idx_t rl[4], ru[4];
            rank_all(f, vl, rl);
            rank_all(f, vu, ru);
            probes += 2;
            step_from_ranks(f, pattern_at(rd, L, kind, d + 1), vl, vu, rl, ru, l[q], u[q], ll[q], uu[q]);
            alive[q] = live(kind, l[q], u[q]);
        }
        ++d;
    }
    while (d < L && (alive[0] || alive[1])) {
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!alive[q]) continue;
            const int kind = q ? k1 : k0;
            const FmView& f = fm[walked_index(kind)];
            const idx_t vl = l[q], vu = u[q] + 1;
            idx_t rl[4], ru[4];
            rank_all(f, vl, rl);
            rank_all(f, vu, ru);
            probes += 2;
            // (#$ in [l, u]) - 1.  The reference also appends the zero-$ case (`tmp >= 0` is
            // always true, src/string_graph.c:229) with remaining size 0; such an entry is never
            // extended, and level 0 never runs the emission check (its max length plus level 0
            // cannot reach L), so it can never contribute and is not stored.
            const idx_t tmp = (vu - (ru[0] + ru[1] + ru[2] + ru[3])) - (vl - (rl[0] + rl[1] + rl[2] + rl[3])) - 1;
            if (tmp + 1 != 0) slots.set(q, n[q]++, ll[q], ll[q] + tmp, pack_meta(d, kind));
            olp = int32_t(uint32_t(olp) + uint32_t(tmp + 1));
            step_from_ranks(f, pattern_at(rd, L, kind, d + 1), vl, vu, rl, ru, l[q], u[q], ll[q], uu[q]);
            alive[q] = live(kind, l[q], u[q]);
        }
        ++d;
    }
}

// One side's candidates into the thread's stack: kind k0 then k1, the reference's order.
__device__ __forceinline__ int side_candidates(const SearchArgs& A, const FmView* fm, const ReadView& rd, idx_t self,
                                               int k0, int k1, Cand* stk, int cap, int& n_out, int32_t& olp,
                                               Tally& probes) {
    const int M = A.L - A.t;
    if (2 * M > cap) return OVF_STACK;
    int n[2];
    chain_pair(A, fm, rd, k0, k1, n, olp, probes, SlotsStack{stk, M});
    for (int i = 0; i < n[1]; ++i) stk[n[0] + i] = stk[M + i];
    n_out = n[0] + n[1];
    return OVF_NONE;
}

__device__ __forceinline__ int cand_index(int type) { return (type == PQ_FB || type == PQ_BB) ? 1 : 0; }

// extract_fw_edges / extract_bw_edges as an explicit DFS over stk[0, n0).  On entering a level the
// emission check runs as in the reference; then all four extension sets are computed at once
// from one pair of block loads per interval (the reference re-probes the same two blocks for
// every base) and stored side by side; the DFS then descends into them in base order A, C, G, T.
// Computing an extension the reference skips (its remaining-size counter reached zero) only
// finds it empty, so the sets are the reference's.
__device__ __forceinline__ int reduce_side(const SearchArgs& A, const FmView* fm, idx_t self, Cand* stk, int cap,
                                           int n0, Frame* fr, int frcap, EdgeRec* eb, int ebcap, int& ne,
                                           int& side_count, Tally& probes) {
    const int L = A.L;
    int level = 0;
    fr[0].pos = 0;
    fr[0].free = uint32_t(n0);
    fr[0].size = uint16_t(n0);
    fr[0].maxlen = 0;
    fr[0].trans = 0;
    bool entering = true;
    while (true) {
        Frame& F = fr[level];
        if (entering) {
            entering = false;
            if (int(F.maxlen) + level == L) {
                bool flag = false;
                for (int i = 0; i < F.size; ++i) {
                    const Cand& c = stk[F.pos + i];
                    if (int(c.len) + level != L) continue;
                    const FmView& fo = fm[cand_index(c.type)];
                    idx_t lll = fo.Cf[0] + rank_dollar(fo, c.ll);
                    idx_t uuu = fo.Cf[0] + rank_dollar(fo, c.uu + 1) - 1;
                    probes += 2;
                    if (lll <= uuu) {
                        probes.add(0, sectors_of(fo.reads_index + lll, size_t(uuu - lll + 1) * sizeof(idx_t)));
                        for (idx_t kk = lll; kk < uuu + 1; ++kk) {
                            idx_t r = __ldg(fo.reads_index + kk);
                            flag = true;
                            if (r != self) {
                                if (side_count + 1 > 65535) return ERR_TOO_MANY;
                                if (ne >= ebcap) return OVF_EDGES;
                                EdgeRec& e = eb[ne++];
                                e.dest = r;
                                e.len = c.len;
                                e.type = c.type;
                                e.trans = F.trans;
                                side_count++;
                            }
                        }
                        break;
                    }
                }
                if (flag) {
                    if (level == 0) return OVF_NONE;
                    --level;
                    continue;
                }
            }
            // all four extension sets from one pair of loads per interval, first in four
            // regions of P slots, then packed back to back in base order
            const int P = F.size;
            const uint32_t cbase = F.free;
            if (int(cbase) + 4 * P > cap) return OVF_STACK;
            int cnt[4] = {0, 0, 0, 0};
            for (int i = 0; i < P; ++i) {
                const Cand c = stk[F.pos + i];
                // remaining size uu - ll + 1 is 0 only for a wrapped [0, all-ones] interval (an
                // empty extension at a zero LF base); the reference keeps it but never extends it
                if (idx_t(c.uu - c.ll + 1) == 0) continue;
                const int o = cand_index(c.type);
                const FmView& f = fm[o];
                idx_t rl[4], ru[4];
                rank_all(f, c.ll, rl);
                rank_all(f, c.uu + 1, ru);
                probes += 2;
                #pragma unroll
                for (int a = 1; a <= 4; ++a) {
                    const int ch = o == 0 ? complement(a) : a;
                    const idx_t ol = pick4(rl, ch), ou = pick4(ru, ch);
                    const idx_t l2 = f.Cf[ch] + ol, u2 = f.Cf[ch] + ou - 1;
                    if (l2 <= u2) {
                        Cand& x = stk[cbase + (a - 1) * P + cnt[a - 1]++];
                        x.ll = l2;
                        x.uu = u2;
                        x.len = c.len;
                        x.type = c.type;
                    }
                }
            }
            int run = cnt[0];
            for (int a = 1; a < 4; ++a) {
                for (int j = 0; j < cnt[a]; ++j) stk[cbase + run + j] = stk[cbase + a * P + j];
                run += cnt[a];
            }
            F.cbase = cbase;
            #pragma unroll
            for (int a = 0; a < 4; ++a) F.csz[a] = uint16_t(cnt[a]);
            F.next_a = 1;
        }
        while (F.next_a <= 4 && F.csz[F.next_a - 1] == 0) F.next_a++;
        if (F.next_a > 4) {
            if (level == 0) return OVF_NONE;
            --level;
            continue;
        }
        const int a = F.next_a++;
        if (level + 1 >= frcap) return OVF_LEVELS;
        Frame& G = fr[level + 1];
        uint32_t before = 0, all = 0;
        #pragma unroll
        for (int b = 0; b < 4; ++b) {
            before += (b < a - 1) ? F.csz[b] : 0;
            all += F.csz[b];
        }
        G.pos = F.cbase + before;
        G.free = F.cbase + all;             // below it: the parent's four sets, still pending
        G.size = F.csz[a - 1];
        int maxl = 0;
        uint32_t tr = 0;
        for (int i = 0; i < G.size; ++i) {
            const Cand& c = stk[G.pos + i];
            tr += uint32_t(c.uu - c.ll + 1);
            maxl = max(maxl, int(c.len));
        }
        G.maxlen = uint16_t(maxl);
        G.trans = int32_t(tr);
        ++level;
        entering = true;
    }
}

__device__ __forceinline__ ReadResult search_read(const SearchArgs& A, const FmView* fm, idx_t self,
                                                  const ReadView& rd, Cand* stk, int cap, Frame* fr, int frcap,
                                                  EdgeRec* eb, int ebcap, Tally& probes) {
    ReadResult R;
    R.status = OVF_NONE;
    R.nB = R.nF = 0;
    R.olpB = R.olpF = 0;
    R.ne = 0;
    int n0 = 0, sc = 0;
    // B side: B-F then B-B candidates, then extract_bw_edges (src/string_graph.c:824-825)
    int s = side_candidates(A, fm, rd, self, PQ_BF, PQ_BB, stk, cap, n0, R.olpB, probes);
    if (s == OVF_NONE && R.olpB != 0)
        s = reduce_side(A, fm, self, stk, cap, n0, fr, frcap, eb, ebcap, R.ne, sc, probes);
    if (s != OVF_NONE) { R.status = s; return R; }
    R.nB = sc;
    // F side: F-B then F-F candidates, then extract_fw_edges (src/string_graph.c:828-829)
    n0 = 0;
    sc = 0;
    s = side_candidates(A, fm, rd, self, PQ_FB, PQ_FF, stk, cap, n0, R.olpF, probes);
    if (s == OVF_NONE && R.olpF != 0)
        s = reduce_side(A, fm, self, stk, cap, n0, fr, frcap, eb, ebcap, R.ne, sc, probes);
    if (s != OVF_NONE) { R.status = s; return R; }
    R.nF = sc;
    return R;
}

__device__ __forceinline__ void load_read(const SearchArgs& A, idx_t r, uint32_t* w, int stride, Tally& probes) {
    const uint8_t* src = A.reads + size_t(r) * A.L;
    probes.add(0, sectors_of(src, size_t(A.L)));
    const int words = (A.L + 15) >> 4;
    for (int i = 0; i < words; ++i) {
        uint32_t v = 0;
        const int j0 = i * 16;
        const int jn = min(16, A.L - j0);
        for (int j = 0; j < jn; ++j) v |= uint32_t(src[j0 + j] - 1) << (2 * j);
        w[i * stride] = v;
    }
}

__device__ __forceinline__ void publish(const SearchOut& O, idx_t r, const ReadResult& R, const EdgeRec* eb) {
    if (R.status != OVF_NONE) {
        O.status[r] = uint8_t(R.status);
        if (R.status != ERR_TOO_MANY) {
            unsigned k = atomicAdd(O.ovf_count, 1u);
            O.ovf_list[k] = r;
        }
        return;
    }
    unsigned long long base = 0;
    if (R.ne) {
        base = atomicAdd(O.e_count, (unsigned long long)R.ne);
        if (base + R.ne > O.e_cap) {
            O.status[r] = OVF_POOL;
            unsigned k = atomicAdd(O.ovf_count, 1u);
            O.ovf_list[k] = r;
            return;
        }
        for (int i = 0; i < R.ne; ++i) {
            O.e_dest[base + i] = eb[i].dest;
            O.e_trans[base + i] = eb[i].trans;
            O.e_len[base + i] = eb[i].len;
            O.e_type[base + i] = eb[i].type;
        }
    }
    O.status[r] = OVF_NONE;
    O.num_B[r] = uint16_t(R.nB);
    O.num_F[r] = uint16_t(R.nF);
    O.olp_B[r] = R.olpB;
    O.olp_F[r] = R.olpF;
    O.edge_src[r] = base;
}

__device__ __forceinline__ void add_probes(const SearchOut& O, const Tally& t) {
    unsigned long long v = t.probes, w = t.sectors;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_down_sync(0xffffffffu, v, o);
        w += __shfl_down_sync(0xffffffffu, w, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (v) atomicAdd(O.probes, v);
        if (w) atomicAdd(O.sectors, w);
    }
}

// ------------------------------------------------------------------------------ fast tier
//
// Phase A: each lane runs the candidate searches of a read (two chains at a time, B side then F
// side); the level-0 candidates of up to kFastQueue reads are packed into the warp's pool.
// Phase B: the (read, side) DFS of extract_*_edges, one a lane, advance together, one level per step;
// a lane whose read is done publishes it (edge-pool reservation, copy, per-read counts) and takes
// the next of the queue.  Each lane owns the control of its read's DFS (frames, emission,
// backtracking); the intervals of all tasks expanding in a step are spread over the lanes, so the
// block loads of up to 32 intervals are in flight together.  The order of the extension sets, the
// first emitting interval and the DFS order of the edges are fixed by entry index (ballots, bit masks
// with population counts, an atomic minimum), never by the order in which lanes happen to run, so
// every edge list is the reference's.
//
// Bound by the latency of the walks' and intervals' blocks (two random sectors each) and by the
// instructions of a step.  1.23 M reads of 100 bases at 30x, 302 M chain steps and 86 M intervals:
// 11.2 ms, 7 of them the chains.  Was 21.2: extensions went through sparse slots and a second pass
// over all four sets of every interval, and a frame was kept at every level (both now only where
// needed: 12.9), with 32 reads at a time in step (15.8 with a queue of 32, 12.5 with 256); five CTAs
// of 96 registers, where six of 80 spill, gave the rest, seven took 16.0, four 12.0.

constexpr int kWarpsPerCta = 4;
constexpr int kTaskCap = 512;       // stack intervals per (read, side) task
constexpr int kTaskFrames = 48;     // DFS frames kept per task (reads with more go to the wide kernel)
constexpr int kPMax = 128;          // intervals of one level of one task

__device__ __forceinline__ int csz_at(uint64_t c4, int i) { return int((c4 >> (16 * i)) & 0xffff); }

// A read of the warp's queue: its level-0 candidates are at `at` in the warp's pool, n[side] of them.
struct FastTask {
    idx_t read;
    uint32_t at;
    int n[2];
};
constexpr int kFastQueue = 128;     // reads a warp walks before it reduces them
constexpr int kFastPool = 4096;     // candidates kept for them (at least one read's most)

// One DFS level of one task (the reference's recursion frame of extract_*_edges).
struct TFrame {
    uint32_t pos;       // first interval of this level in the task's stack
    uint32_t free;      // first stack slot this level may use for its extension sets
    uint32_t cbase;     // first slot of the four extension sets (back to back, A..T)
    int32_t trans;      // sum of this level's interval sizes (path_t.trans of its edges)
    uint16_t size, maxlen;
    uint16_t next_a, level;
    uint64_t csz4;      // sizes of the four sets, 16 bits each (A lowest)
    uint64_t cml4;      // largest overlap length in each set, 16 bits each
    int32_t ctr[4];     // interval-size sum of each set
};

// Shared memory of one warp for the level-synchronous DFS of its 32 tasks (MW 64-bit mask words
// per larger task and base: one bit per interval of a level, up to 64 MW intervals).
template <int MW>
struct MultiSmem {
    unsigned long long mask[32][4][MW];  // extension present, by entry index
    int hit[32];                         // first entry that completes a read with $ rows
    int cml[32][4];
    unsigned ctr[32][4];
    int setoff[32][4];
    int pref[33];
    uint32_t pos[32], cbase[32];
    int lvl[32], chk[32], size[32];
    uint32_t src[32];                    // pool position of a task's level 0
    int list[32];                        // the tasks of up to 32 intervals, in lane order
    uint32_t cnt[32];                    // their four sets' sizes, 8 bits each
};

template <int MW>
__device__ __forceinline__ int popc_words(const unsigned long long* m) {
    int c = 0;
    #pragma unroll
    for (int w = 0; w < MW; ++w) c += __popcll(m[w]);
    return c;
}
// set bits of m below bit i
template <int MW>
__device__ __forceinline__ int popc_below(const unsigned long long* m, int i) {
    int c = 0;
    #pragma unroll
    for (int w = 0; w < MW; ++w) {
        const int lo = 64 * w;
        if (i >= lo + 64) c += __popcll(m[w]);
        else if (i > lo) c += __popcll(m[w] & ((1ull << (i - lo)) - 1));
    }
    return c;
}

// exclusive prefix of v over the warp into pref[0..32] (pref[32] = total), returns the total
__device__ __forceinline__ int warp_prefix(int v, int* pref) {
    const int lane = threadIdx.x & 31;
    int x = v;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    pref[lane] = x - v;
    if (lane == 31) pref[32] = x;
    __syncwarp();
    return pref[32];
}

// task owning flattened item e (pref ascending, pref[32] = total)
__device__ __forceinline__ int owner_of(const int* pref, int e) {
    int lo = 0, hi = 31;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pref[mid] <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ------------------------------------------------------------------------------ sorted reduction
//
// extract_*_edges as a function of the candidate set.  At DFS level j an interval of candidate
// group (kind, d) holds exactly the candidates r' whose next j bases after the overlap -- their
// continuation lambda(r') -- equal the DFS path s: extending the other index's interval by base a
// selects the candidates whose next base is a (the complement on the forward index).  So the DFS
// is a walk over the trie of continuations in base order, and:
//   * it emits at node s exactly when some candidate's continuation is s (its len + level == L),
//     taking the first interval in stack order with that length -- the group of the side's first
//     kind if it has a candidate there, else the second kind's -- and its reads (in row order,
//     i.e. ascending read id, the read itself left out), with path_t.trans = the number of
//     candidates whose continuation starts with s (the frame's interval sizes summed);
//   * an emission ends the branch, so a candidate whose continuation has another candidate's as a
//     proper prefix is never reached.
// Below, each candidate's continuation (L - d <= 256 bases) is read from the packed text -- the
// forward text from r' * L + d for candidates on the backward index, the complemented backward
// text there for candidates on the forward index -- and the emitted edges are ordered by
// continuation, then read id: the DFS order.  No FM-index step is taken.

constexpr int kRedMax = 64;          // candidates of one (read, side) reduced this way
// candidate i of lane l of a warp sits at slot 32 i + l of the warp's arrays, so that the lanes of a
// warp, each reducing its own read in step with the others, load consecutive words
constexpr int kRedStride = 32;
constexpr int kLamWords = 8;         // continuations up to 256 bases (L - t <= 256)

// continuation words the kernels are built for: 2 (L - t <= 64) or kLamWords
__host__ __device__ constexpr int lam_words(int M) { return M <= 64 ? 2 : kLamWords; }

// word w of the continuation of candidate r' at overlap d (32 w < L - d)
__device__ __forceinline__ uint64_t continuation_word(const SearchArgs& A, int type, idx_t rp, int d, int w) {
    const bool fwd = cand_index(type) == 1;
    const int left = A.L - d - 32 * w;
    const uint64_t x = text_window(A.fm[fwd ? 0 : 1].pk, size_t(rp) * A.L + size_t(d) + 32 * size_t(w));
    return (fwd ? x : ~x) & top_mask(left < 32 ? left : 32);
}

// continuation of candidate r' at overlap d: L - d bases (at most 32 W) in ceil((L - d) / 32)
// words, first base in the top bits, zero past the end; word w at out[w * plane]
// (returns the 32-byte sectors of packed text it loaded)
template <int W>
__device__ __forceinline__ uint32_t continuation(const SearchArgs& A, int type, idx_t rp, int d, uint64_t* out,
                                                 size_t plane) {
    const int len = A.L - d;
    #pragma unroll
    for (int w = 0; w < W; ++w) {
        if (32 * w >= len) break;
        out[w * plane] = continuation_word(A, type, rp, d, w);
    }
    return len > 0 ? base_sectors(size_t(rp) * A.L + size_t(d), len) : 0;
}

// The candidates of one (read, side) as the reduction sees them: read id, (overlap, kind) and
// continuation words of candidate i, in the warp's global scratch.  (The first 8 or 16 of a read in
// shared memory instead: 12.0 and 8.9 ms against 7.2 on 5.4 M reads, for want of L1 and of warps.)
struct Cands {
    const WarpScratch& S;
    size_t red;
    __device__ __forceinline__ size_t at(int i) const { return red + size_t(i) * kRedStride; }
    __device__ __forceinline__ idx_t id(int i) const { return S.r_id[at(i)]; }
    __device__ __forceinline__ uint32_t meta(int i) const { return S.r_meta[at(i)]; }
    __device__ __forceinline__ uint64_t word(int i, int w) const { return S.r_k[w * S.r_plane + at(i)]; }
};
// order of candidates i and j, whose continuations (la and lb bases) are equal or not prefixes of
// one another: their first differing base, else equal
template <int W>
__device__ __forceinline__ int cmp_cont(const Cands& C, int i, int la, int j, int lb) {
    const int n = la < lb ? la : lb;
    #pragma unroll
    for (int w = 0; w < W; ++w) {
        if (32 * w >= n) break;
        const uint64_t x = C.word(i, w), y = C.word(j, w);
        if (x != y) return x < y ? -1 : 1;
    }
    return la == lb ? 0 : (la < lb ? -1 : 1);
}

template <int W>
__device__ __forceinline__ int reduce_gathered(int L, const WarpScratch& S, idx_t self, int side, size_t red, int m,
                                               size_t eb, int estride, int& ne, int& count);

// Edges of one side of one read from its level-0 candidate groups (na of the first kind, then
// n0 - na of the second) in the candidate scratch at `cand`; per-lane scratch at `red`.
template <int W>
__device__ __forceinline__ int reduce_sorted(const SearchArgs& A, const WarpScratch& S, idx_t self, int side,
                                             size_t cand, int n0, size_t red, size_t eb, int& ne,
                                             int& count, Tally& probes) {
    const int L = A.L;
    int m = 0;
    for (int g = 0; g < n0; ++g) {
        const idx_t ll = S.p_ll[cand + g], uu = S.p_uu[cand + g];
        const uint32_t mt = S.p_meta[cand + g];
        const int d = meta_len(mt), type = meta_type(mt);
        const FmView& fb = A.fm[cand_index(type)];
        for (idx_t row = ll; row <= uu; ++row) {
            const idx_t p = __ldg(fb.sa + row);
            const idx_t rp = read_of(p, A.dl);
            const size_t q = red + size_t(m) * kRedStride;
            const uint32_t sec = continuation<W>(A, type, rp, d, S.r_k + q, S.r_plane);
            S.r_id[q] = rp;
            S.r_meta[q] = mt;
            probes.add(2, 1 + sec);
            ++m;
        }
    }
    return reduce_gathered<W>(L, S, self, side, red, m, eb, 1, ne, count);
}

// The reduction of reduce_sorted over m <= 64 gathered candidates; `red` is the lane's column of the
// warp's scratch (kRedStride).  Emitted edges go to the edge scratch at eb + estride ne, in DFS order.
//
// In rounds: the shortest continuation left, s, has no proper prefix among the others, so its class
// -- the candidates left whose continuation starts with s -- is emitted where it equals s and covered
// where it goes on, and trans is the class's size: a candidate of an earlier class starts with a
// prefix of s only if s itself did.  Most candidates of a read continue one genome locus, so one or
// two rounds, each a test a candidate, take the place of a test for every pair (the reduction of 5.4
// M reads at 20x took 3.5 ms by pairs).
template <int W>
__device__ __forceinline__ int reduce_gathered(int L, const WarpScratch& S, idx_t self, int side, size_t red, int m,
                                               size_t eb, int estride, int& ne, int& count) {
    const Cands C{S, red};
    const int first_kind = side ? PQ_FB : PQ_BF;
    auto at = [&](int i) { return red + size_t(i) * kRedStride; };
    auto bit = [](int i) { return 1ull << i; };
    int nemit = 0;
    unsigned long long left = m >= 64 ? ~0ull : bit(m) - 1;
    while (left) {
        int ls = 1 << 30, is = 0;
        for (unsigned long long x = left; x; x &= x - 1) {
            const int c = __ffsll((long long)x) - 1;
            const int lc = L - meta_len(C.meta(c));
            if (lc < ls) {
                ls = lc;
                is = c;
            }
        }
        uint64_t ks[W];
        #pragma unroll
        for (int w = 0; w < W; ++w) ks[w] = 32 * w < ls ? C.word(is, w) : 0;
        unsigned long long cls = 0, equal = 0;
        bool first_same = false;
        for (unsigned long long x = left; x; x &= x - 1) {
            const int c = __ffsll((long long)x) - 1;
            const uint32_t mc = C.meta(c);
            bool same = true;
            #pragma unroll
            for (int w = 0; w < W; ++w) {
                const int rest = ls - 32 * w;
                if (rest > 0 && same) same = ((C.word(c, w) ^ ks[w]) & top_mask(rest < 32 ? rest : 32)) == 0;
            }
            if (!same) continue;
            cls |= bit(c);
            if (L - meta_len(mc) == ls) {
                equal |= bit(c);
                first_same = first_same || meta_type(mc) == first_kind;
            }
        }
        left &= ~cls;
        const uint32_t trans = uint32_t(__popcll(cls));
        for (; equal; equal &= equal - 1) {
            const int c = __ffsll((long long)equal) - 1;
            if (C.id(c) == self || (first_same && meta_type(C.meta(c)) != first_kind)) continue;
            S.r_emit[at(nemit++)] = uint32_t(c) | (trans << 16);
        }
    }
    // DFS order: continuation, then read id (insertion sort; a handful of edges)
    for (int i = 1; i < nemit; ++i) {
        const uint32_t x = S.r_emit[at(i)];
        const int cx = int(x & 0xffff);
        const int lx = L - meta_len(C.meta(cx));
        const idx_t xi = C.id(cx);
        int j = i - 1;
        while (j >= 0) {
            const int cy = int(S.r_emit[at(j)] & 0xffff);
            const int o = cmp_cont<W>(C, cy, L - meta_len(C.meta(cy)), cx, lx);
            const bool greater = o != 0 ? o > 0 : C.id(cy) > xi;
            if (!greater) break;
            S.r_emit[at(j + 1)] = S.r_emit[at(j)];
            --j;
        }
        S.r_emit[at(j + 1)] = x;
    }
    for (int i = 0; i < nemit; ++i) {
        const uint32_t x = S.r_emit[at(i)];
        const int c = int(x & 0xffff);
        if (ne >= S.ebcap) return OVF_EDGES;
        const size_t q = eb + size_t(ne) * estride;
        S.e_dest[q] = C.id(c);
        S.e_trans[q] = int32_t(x >> 16);
        S.e_meta[q] = C.meta(c);
        ++ne;
    }
    count = nemit;
    return OVF_NONE;
}

// ------------------------------------------------------------------------ lean tier: candidate scan
//
// The interval scan already yields every candidate of a side with its read id and overlap -- row
// (r', o) of I_t is a candidate at depth t + o -- and its continuation is the rest of r' after the
// overlap: the walked index's text right after the matched pattern, at the row's text position
// plus t (complemented for the kinds walked on the backward index, B-F and F-F).  So the lean tier
// gathers each side's candidates for reduce_gathered straight from the scan.

// Rows [first, end) of each chain's index to check for the patterns P0 and P1 of one side's chains,
// all rows that start with their first t bases among them; false when the scan does not apply to this
// read (a depth-t interval of more than kScanMax rows, or a learned window that missed): the block
// tier then redoes it.

// The window of the learned index, narrowed to I_t (seed mode 2).
__device__ __forceinline__ bool learned_rows(const SearchArgs& A, const FmView* f0, const FmView* f1,
                                             const uint64_t (&P0)[kScanWords], const uint64_t (&P1)[kScanWords],
                                             idx_t (&first)[2], idx_t (&end)[2], Tally& probes) {
    const int tb = A.t < 32 * kScanWords ? A.t : 32 * kScanWords;
    const FmView* fq[2] = {f0, f1};
    idx_t lo[2], hi[2];
    #pragma unroll
    for (int q = 0; q < 2; ++q) {
        const LearnedView& v = fq[q]->lx;
        const uint32_t K = uint32_t((q ? P1 : P0)[0] >> 32);
        const int sg = lx_segment(v, K);
        const long long pr = lx_predict(v, sg, K);
        const long long b0 = (long long)__ldg(v.base + sg), b1 = (long long)__ldg(v.base + sg + 1);
        const long long a = pr - (long long)__ldg(v.err + 2 * sg), b = pr + (long long)__ldg(v.err + 2 * sg + 1);
        lo[q] = idx_t(a > b0 ? a : b0);
        hi[q] = idx_t(b < b1 ? b : b1);
        if (hi[q] < lo[q]) hi[q] = lo[q];
    }
    sa_bounds2(f0, f1, A.dl, P0, P1, tb, lo, hi, first, end, probes);
    // The window holds the answer for every key present in the index; for any other key it
    // is checked: the rows just outside the window must not start with P_t.
    const idx_t n_rows = A.num_reads * idx_t(A.L);
    bool ok = true;
    #pragma unroll
    for (int q = 0; q < 2; ++q) {
        const FmView& fa = *fq[q];
        const uint64_t (&P)[kScanWords] = q ? P1 : P0;
        if (first[q] == lo[q] && lo[q] > 0) {
            const idx_t p = __ldg(fa.sa + lo[q] - 1);
            ok = ok && cmp_row(fa.pk, p, suffix_len(p, A.dl), P, tb) < 0;
            probes.add(2, 1 + cmp_sectors(fa.pk, p));
        }
        if (end[q] == hi[q] && hi[q] < n_rows) {
            const idx_t p = __ldg(fa.sa + hi[q]);
            ok = ok && cmp_row(fa.pk, p, suffix_len(p, A.dl), P, tb) > 0;
            probes.add(2, 1 + cmp_sectors(fa.pk, p));
        }
    }
    if (!ok) atomicAdd(A.lx_misses, 1ull);
    return ok && end[0] - first[0] <= idx_t(kScanMax) && end[1] - first[1] <= idx_t(kScanMax);
}

// Of the rows [lo, hi) of a k-mer, those that go on with the next bases of its pattern, whose first
// 32 bases are `word`.  Up to 64 rows are all read, 8 to a 16-byte load and independent of one
// another, and compared two to a word (kx values are below 2^15, which leaves each half a guard
// bit); a binary search would wait for three or four dependent sectors (3.5 ms against 1.2 on 5.4 M
// reads of 44 rows a k-mer).  More rows are searched.
__device__ __forceinline__ void narrow_rows(const FmView& f, int k, int t, uint64_t word, idx_t& lo, idx_t& hi, Tally& probes) {
    const int x = f.kx_bases < t - k ? f.kx_bases : t - k;
    if (x <= 0 || hi - lo <= 4) return;
    const int drop = 2 * (f.kx_bases - x);
    const uint32_t want = uint32_t(word << (2 * k) >> (64 - 2 * x));
    const uint32_t from = want << drop, past = (want + 1) << drop;          // the values of the rows wanted
    if (hi - lo <= 64) {
        const idx_t base = lo & ~idx_t(7);
        const int chunks = int(hi - base + 7) >> 3, skip = int(lo - base), held = int(hi - base) - 8 * (chunks - 1);
        const uint4* v = reinterpret_cast<const uint4*>(f.kx + base);
        // a chunk's rows 0, 2, 4, 6 in bits 0..3 and 1, 3, 5, 7 in bits 16..19: those from `skip` on
        // in the first, the first `held` in the last
        const uint32_t head = ((0xfu << ((skip + 1) >> 1)) & 0xfu) | (((0xfu << (skip >> 1)) & 0xfu) << 16);
        const uint32_t tail = ((1u << ((held + 1) >> 1)) - 1u) | (((1u << (held >> 1)) - 1u) << 16);
        const uint32_t from2 = from * 0x10001u, past2 = past * 0x10001u;
        constexpr uint32_t H = 0x80008000u;
        int below = 0, upto = 0;
        #pragma unroll 3
        for (int c = 0; c < chunks; ++c) {
            const uint4 q = __ldg(v + c);
            const uint32_t in = (c ? 0xf000fu : head) & (c + 1 < chunks ? 0xf000fu : tail);
            auto less = [&](uint32_t w, uint32_t than) { return ~((w | H) - than) & H; };
            auto rows = [&](uint32_t than) {
                return (less(q.x, than) >> 15) | (less(q.y, than) >> 14) | (less(q.z, than) >> 13) | (less(q.w, than) >> 12);
            };
            below += __popc(rows(from2) & in);
            upto += __popc(rows(past2) & in);
        }
        probes.add(0, uint32_t(chunks + 1) / 2);
        hi = lo + idx_t(upto);
        lo += idx_t(below);
        return;
    }
    idx_t first = lo, b = hi;
    while (first < b) {
        const idx_t m = first + (b - first) / 2;
        if (__ldg(f.kx + m) < from) first = m + 1;
        else b = m;
        probes.add(0, 1);
    }
    idx_t end = first;
    b = hi;
    while (end < b) {
        const idx_t m = end + (b - end) / 2;
        if (__ldg(f.kx + m) < past) end = m + 1;
        else b = m;
        probes.add(0, 1);
    }
    lo = first;
    hi = end;
}

// warp-cooperative copy of one batch description into shared memory
__device__ __forceinline__ void load_batch(SearchBatch& dst, const SearchBatch* src, int lane) {
    static_assert(sizeof(SearchBatch) % 4 == 0, "batch description is copied in 32-bit words");
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
    for (int i = lane; i < int(sizeof(SearchBatch) / 4); i += 32) d[i] = s[i];
    __syncwarp();
}

// A lane's read is done: its edges (eb .. eb + ne: B side, then F side) to the pool and its counts, or
// the next tier's list.
__device__ __forceinline__ void publish_lane(const SearchOut& O, const WarpScratch& S, idx_t r, int status, size_t eb, int ne,
                                             int count_b, int count_f) {
    unsigned long long base = 0;
    if (status == OVF_NONE && ne) {
        base = atomicAdd(O.e_count, (unsigned long long)ne);
        if (base + ne > O.e_cap) status = OVF_POOL;
    }
    O.status[r] = uint8_t(status);
    if (status != OVF_NONE) {
        if (status != ERR_TOO_MANY) {
            const unsigned k = atomicAdd(O.ovf_count, 1u);
            O.ovf_list[k] = r;
        }
        return;
    }
    for (int e = 0; e < ne; ++e) {
        const uint32_t mt = S.e_meta[eb + e];
        O.e_dest[base + e] = S.e_dest[eb + e];
        O.e_trans[base + e] = S.e_trans[eb + e];
        O.e_len[base + e] = uint16_t(meta_len(mt));
        O.e_type[base + e] = uint8_t(meta_type(mt));
    }
    O.num_B[r] = uint16_t(count_b);
    O.num_F[r] = uint16_t(count_f);
    O.edge_src[r] = base;
}

// Without a queue (Q.count == 0) the kernel searches the one read set of (A0, O0), warp w taking
// groups of 32 reads w, w + #warps, ...  With a queue, each warp takes the next item (a batch and
// a group of its reads) from a shared counter until the queue is empty; the batch's description
// (index pair, L, t, outputs) is loaded into the warp's shared memory when it changes.
template <int W, int CAP, int FRAMES, int PMAX>
__global__ void __launch_bounds__(128, 5) k_search_fast(SearchArgs A0, SearchOut O0, WarpScratch S, SearchQueue Q) {
    constexpr int MW = PMAX / 64;
    extern __shared__ uint32_t s_reads[];
    __shared__ SearchBatch s_b[kWarpsPerCta];
    __shared__ MultiSmem<MW> s_ms[kWarpsPerCta];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const size_t gw = size_t(blockIdx.x) * kWarpsPerCta + wid;
    const size_t nw = size_t(gridDim.x) * kWarpsPerCta;
    SearchBatch& B = s_b[wid];
    const SearchArgs& A = B.a;
    const SearchOut& O = B.o;
    if (Q.count == 0) {
        if (lane == 0) {
            B.a = A0;
            B.o = O0;
        }
        __syncwarp();
    }
    MultiSmem<MW>& sm = s_ms[wid];
    const size_t cbase_w = gw * 32 * 4 * size_t(S.mstride);    // level-0 candidates of 32 reads
    const size_t pbase_w = gw * size_t(S.pool);                // and of the queued reads, packed
    FastTask* const queue = S.queue + gw * kFastQueue;
    const size_t ebase_w = gw * 32 * size_t(S.ebcap);          // edge slots of this warp
    const size_t tbase_w = gw * 32 * size_t(CAP);         // task stacks
    const size_t xbase_w = gw * 32 * 4 * size_t(PMAX);        // sparse extension slots
    const size_t mbase_w = gw * 32 * size_t(PMAX);            // emission bounds
    const size_t rbase_w = gw * 32 * size_t(kRedMax);          // sorted-reduction candidates
    TFrame* const frw = S.frames + gw * 32 * FRAMES;
    Tally probes;
    int cur = -1;
    // reads of the current batch (or of the list of reads handed over by the lean tier)
    const size_t list_n = Q.read_list ? size_t(*Q.list_count) : 0;
    while (true) {
        size_t group = gw, gend = 0, step = nw;
        if (Q.count) {
            unsigned it = 0;
            if (lane == 0) it = atomicAdd(Q.next, 1u);
            it = __shfl_sync(0xffffffffu, it, 0);
            if (it >= Q.count) break;
            const int b = int(Q.item_batch[it]);
            group = Q.item_group[it];
            gend = group + Q.groups_per_item;
            step = 1;
            if (b != cur) {
                if (cur >= 0) add_probes(O, probes);
                probes = Tally{};
                __syncwarp();
                load_batch(B, Q.batches + b, lane);
                cur = b;
            }
        }
        const size_t n_items = Q.read_list ? list_n : size_t(A.num_reads);
        const size_t groups = (n_items + Q.per - 1) / Q.per;
        if (!Q.count || gend > groups) gend = groups;
        const int M = A.L - A.t;
        const int L = A.L;
        bool pend = false;          // this lane's read of the last group walked waits for room in the queue
        idx_t pr = 0;
        int pn[4] = {0, 0, 0, 0};
        while (true) {
        // ---- phase A
        int nq = 0, used = 0;
        while (true) {
            if (!__any_sync(0xffffffffu, pend)) {
                if (group >= gend || nq + 32 > kFastQueue) break;
                const size_t item = group * Q.per + lane;
                pend = unsigned(lane) < Q.per && item < n_items;
                group += step;
                if (pend) {
                    pr = Q.read_list ? Q.read_list[item] : idx_t(item);
                    load_read(A, pr, s_reads + threadIdx.x, blockDim.x, probes);
                    const ReadView rd{s_reads + threadIdx.x, int(blockDim.x)};
                    const size_t cb = cbase_w + size_t(lane);
                    int n[2];
                    int32_t olp = 0;
                    chain_pair(A, A.fm, rd, PQ_BF, PQ_BB, n, olp, probes, SlotsFast{S.c_ll, S.c_uu, S.c_meta, cb, M});
                    O.olp_B[pr] = olp;
                    pn[0] = n[0];
                    pn[1] = n[1];
                    olp = 0;
                    chain_pair(A, A.fm, rd, PQ_FB, PQ_FF, n, olp, probes,
                               SlotsFast{S.c_ll, S.c_uu, S.c_meta, cb + size_t(2 * M) * 32, M});
                    O.olp_F[pr] = olp;
                    pn[2] = n[0];
                    pn[3] = n[1];
                }
                __syncwarp();
            }
            const int mine = pend ? pn[0] + pn[1] + pn[2] + pn[3] : 0;
            int incl = mine;
            #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const bool fits = pend && used + incl <= S.pool;
            const unsigned take = __ballot_sync(0xffffffffu, fits);
            if (!take) break;
            if (fits) {
                uint32_t to = uint32_t(used + incl - mine);
                queue[nq + __popc(take & ((1u << lane) - 1u))] = FastTask{pr, to, {pn[0] + pn[1], pn[2] + pn[3]}};
                #pragma unroll
                for (int q = 0; q < 4; ++q)
                    for (int i = 0; i < pn[q]; ++i, ++to) {
                        const size_t src = cbase_w + (size_t(q) * M + i) * 32 + size_t(lane);
                        S.p_ll[pbase_w + to] = S.c_ll[src];
                        S.p_uu[pbase_w + to] = S.c_uu[src];
                        S.p_meta[pbase_w + to] = S.c_meta[src];
                    }
                pend = false;
            }
            nq += __popc(take);
            used += __shfl_sync(0xffffffffu, incl, 31 - __clz(int(take)));
            __syncwarp();
            if (__any_sync(0xffffffffu, pend)) break;
        }
        if (!nq) break;
        // ---- phase B
        int next_q = 0, qi = 0, side = 0;
        bool busy = false, active = false, entering = false;
        idx_t self = 0;
        int status = OVF_NONE, ne = 0, count_b = 0, level = 0, sp = 0, sc = 0;
        const size_t tb = tbase_w + size_t(lane) * CAP;    // this lane's task stack
        TFrame* const fr = frw + lane * FRAMES;
        const size_t eb = ebase_w + size_t(lane) * S.ebcap;
        TFrame F{};
        while (true) {
            // (0) lanes without a task take the next: the read's other side, or the next read's first
            bool fresh = false;
            uint32_t src = 0;
            while (__any_sync(0xffffffffu, (busy && !active) || (!busy && next_q < nq))) {
                bool setup = false;
                if (busy && !active) {
                    if (side == 0 && status == OVF_NONE) {
                        count_b = sc;
                        side = 1;
                        setup = true;
                    } else {
                        publish_lane(O, S, self, status, eb, ne, side ? count_b : sc, side ? sc : 0);
                        busy = false;
                    }
                }
                const unsigned idle = __ballot_sync(0xffffffffu, !busy);
                if (!busy) {
                    qi = next_q + __popc(idle & ((1u << lane) - 1u));
                    if (qi < nq) {
                        self = queue[qi].read;
                        busy = setup = true;
                        side = 0;
                        status = OVF_NONE;
                        ne = 0;
                    }
                }
                next_q = min(nq, next_q + __popc(idle));
                if (setup) {
                    const FastTask task = queue[qi];
                    const int n0 = side ? task.n[1] : task.n[0];
                    const int32_t olp = side ? O.olp_F[self] : O.olp_B[self];
                    src = task.at + uint32_t(side ? task.n[0] : 0);
                    sc = 0;
                    active = olp != 0;                                  // src/string_graph.c:824, 828
                    if (active && A.sorted_reduce && olp <= kRedMax) {
                        const int st = reduce_sorted<W>(A, S, self, side, pbase_w + src, n0, rbase_w + lane, eb, ne, sc, probes);
                        if (st != OVF_NONE) status = st;
                        active = false;
                    } else if (active && n0 > Q.dfs_max) {
                        status = OVF_STACK;
                        active = false;
                    }
                    fresh = active;
                    F = TFrame{};
                    F.free = uint32_t(n0);
                    F.size = uint16_t(n0);
                    F.next_a = 1;
                    entering = true;
                    level = sp = 0;
                }
            }
            if (!__any_sync(0xffffffffu, busy)) break;
            // level 0: kind-0 candidates then kind-1 candidates
            if (__any_sync(0xffffffffu, fresh)) {
                sm.src[lane] = src;
                const int tot0 = warp_prefix(fresh ? int(F.size) : 0, sm.pref);
                for (int e = lane; e < tot0; e += 32) {
                    const int j = owner_of(sm.pref, e);
                    const int i = e - sm.pref[j];
                    const size_t from = pbase_w + sm.src[j] + i, dst = tbase_w + size_t(j) * CAP + i;
                    S.t_ll[dst] = S.p_ll[from];
                    S.t_uu[dst] = S.p_uu[from];
                    S.t_meta[dst] = S.p_meta[from];
                }
                __syncwarp();
            }
            {
                // (1) own control: backtrack / descend until this task needs an expansion.  A frame
                // is kept only while sets of it remain: the last one is entered in its place.
                if (active && !entering) {
                    while (true) {
                        int a = int(F.next_a);
                        while (a <= 4 && csz_at(F.csz4, a - 1) == 0) ++a;
                        if (a > 4) {
                            if (sp == 0) { active = false; break; }
                            F = fr[--sp];
                            level = F.level;
                            continue;
                        }
                        uint32_t before = 0, all = 0;
                        #pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            before += (b < a - 1) ? csz_at(F.csz4, b) : 0;
                            all += csz_at(F.csz4, b);
                        }
                        if (all > before + csz_at(F.csz4, a - 1)) {
                            if (sp >= FRAMES) { status = OVF_LEVELS; active = false; break; }
                            F.next_a = uint16_t(a + 1);
                            F.level = uint16_t(level);
                            fr[sp++] = F;
                        }
                        F.size = uint16_t(csz_at(F.csz4, a - 1));
                        F.maxlen = uint16_t(csz_at(F.cml4, a - 1));
                        F.trans = a == 1 ? F.ctr[0] : (a == 2 ? F.ctr[1] : (a == 3 ? F.ctr[2] : F.ctr[3]));
                        F.pos = F.cbase + before;
                        F.free = F.cbase + all;      // below it: the parent's four sets, still pending
                        F.next_a = 1;
                        F.csz4 = 0;
                        ++level;
                        entering = true;
                        break;
                    }
                }
                const bool expand = active && entering;
                if (expand && F.size > PMAX) { status = OVF_STACK; active = false; }
                const bool go = active && entering;
                const bool narrow = go && F.size > 0 && F.size <= 32;
                const bool chk = int(F.maxlen) + level == L;
                sm.hit[lane] = 0x7fffffff;
                sm.cnt[lane] = 0;
                #pragma unroll
                for (int a = 0; a < 4; ++a) {
                    sm.cml[lane][a] = 0;
                    sm.ctr[lane][a] = 0;
                }
                // (2) every interval of every expanding task: one pair of block loads serves the
                // emission check and the four extensions.  Tasks of up to 32 intervals, as many
                // whole ones as fit the lanes at a time: their sets are counted by ballots and
                // written where they belong.
                {
                    const int size = narrow ? int(F.size) : 0;
                    int end = size;
                    #pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, end, o);
                        if (lane >= o) end += y;
                    }
                    const int total = __shfl_sync(0xffffffffu, end, 31), mine = end - size;
                    const unsigned all = __ballot_sync(0xffffffffu, narrow);
                    if (narrow) sm.list[__popc(all & ((1u << lane) - 1u))] = lane;
                    __syncwarp();
                    for (int base = 0, first = 0; base < total;) {
                        const bool in = narrow && mine >= base && end <= base + 32;
                        const unsigned starts = __reduce_or_sync(0xffffffffu, in ? 1u << (mine - base) : 0u);
                        const unsigned tasks = __ballot_sync(0xffffffffu, in);
                        const int n = __shfl_sync(0xffffffffu, end, 31 - __clz(int(tasks))) - base;
                        const unsigned at = starts & (0xffffffffu >> (31 - lane));
                        const int s = 31 - __clz(int(at)), j = sm.list[first + __popc(at) - 1];
                        const unsigned over = starts & (0xfffffffeu << lane);
                        const int e = over ? __ffs(int(over)) - 1 : n;
                        const unsigned seg = (e < 32 ? (1u << e) - 1u : 0xffffffffu) & (0xffffffffu << s);
                        const uint32_t pos = __shfl_sync(0xffffffffu, F.pos, j), free = __shfl_sync(0xffffffffu, F.free, j);
                        const int lc = __shfl_sync(0xffffffffu, chk ? level : -1, j);
                        const size_t tj = tbase_w + size_t(j) * CAP;
                        bool emits = false;
                        idx_t lo[4], hi[4], ea = 0, eb2 = 0;
                        unsigned has = 0;
                        uint32_t m = 0;
                        if (lane < n) {
                            const size_t from = tj + pos + (lane - s);
                            const idx_t cl = S.t_ll[from], cu = S.t_uu[from];
                            m = S.t_meta[from];
                            const bool ext = idx_t(cu - cl + 1) != 0;   // wrapped [0, all-ones]: kept, never extended
                            const bool ends = lc >= 0 && meta_len(m) + lc == L;
                            const int o = cand_index(meta_type(m));
                            const FmView& f = A.fm[o];
                            idx_t rl[4] = {0, 0, 0, 0}, ru[4] = {0, 0, 0, 0};
                            if (ext || ends) {
                                rank_all(f, cl, rl);
                                rank_all(f, cu + 1, ru);
                                probes += 2;
                            }
                            if (ends) {
                                ea = f.Cf[0] + (cl - (rl[0] + rl[1] + rl[2] + rl[3]));
                                eb2 = f.Cf[0] + ((cu + 1) - (ru[0] + ru[1] + ru[2] + ru[3])) - 1;
                                emits = ea <= eb2;
                            }
                            if (ext) {
                                #pragma unroll
                                for (int a = 1; a <= 4; ++a) {
                                    const int ch = o == 0 ? complement(a) : a;
                                    lo[a - 1] = f.Cf[ch] + pick4(rl, ch);
                                    hi[a - 1] = f.Cf[ch] + pick4(ru, ch) - 1;
                                    has |= lo[a - 1] <= hi[a - 1] ? 1u << (a - 1) : 0u;
                                }
                            }
                        }
                        const unsigned em = __ballot_sync(0xffffffffu, emits) & seg;
                        if (emits && !(em & ((1u << lane) - 1u))) {
                            const size_t me = mbase_w + size_t(j) * PMAX + (lane - s);
                            S.em_l[me] = ea;
                            S.em_u[me] = eb2;
                            sm.hit[j] = lane - s;
                        }
                        unsigned to = free, cnt = 0, b[4];
                        #pragma unroll
                        for (int a = 0; a < 4; ++a) {
                            b[a] = __ballot_sync(0xffffffffu, (has >> a) & 1u) & seg;
                            cnt |= unsigned(__popc(b[a])) << (8 * a);
                        }
                        if (lane < n) {
                            if (lane == s) sm.cnt[j] = cnt;
                            const bool room = free + __popc(b[0]) + __popc(b[1]) + __popc(b[2]) + __popc(b[3]) <= unsigned(CAP);
                            #pragma unroll
                            for (int a = 0; a < 4; ++a) {
                                if (((has >> a) & 1u) && room) {
                                    const size_t x = tj + to + __popc(b[a] & ((1u << lane) - 1u));
                                    S.t_ll[x] = lo[a];
                                    S.t_uu[x] = hi[a];
                                    S.t_meta[x] = m;
                                    atomicMax(&sm.cml[j][a], meta_len(m));
                                    atomicAdd(&sm.ctr[j][a], unsigned(hi[a] - lo[a] + 1));
                                }
                                to += __popc(b[a]);
                            }
                        }
                        first += __popc(tasks);
                        base += n;
                    }
                }
                // larger tasks: the intervals of all of them one after the other, extensions by
                // entry first, packed below
                const bool broad = go && F.size > 32, any_broad = __any_sync(0xffffffffu, broad);
                if (any_broad) {
                    sm.size[lane] = broad ? int(F.size) : 0;
                    sm.pos[lane] = F.pos;
                    sm.lvl[lane] = level;
                    sm.chk[lane] = chk;
                    #pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        #pragma unroll
                        for (int w = 0; w < MW; ++w) sm.mask[lane][a][w] = 0;
                    }
                const int tot = warp_prefix(broad ? int(F.size) : 0, sm.pref);
                for (int e = lane; e < tot; e += 32) {
                    const int j = owner_of(sm.pref, e);
                    const int i = e - sm.pref[j];
                    const size_t tj = tbase_w + size_t(j) * CAP + sm.pos[j] + i;
                    const idx_t cl = S.t_ll[tj], cu = S.t_uu[tj];
                    const uint32_t m = S.t_meta[tj];
                    const bool ext = idx_t(cu - cl + 1) != 0;   // wrapped [0, all-ones]: kept, never extended
                    const bool ends = sm.chk[j] && meta_len(m) + sm.lvl[j] == L;
                    const int o = cand_index(meta_type(m));
                    const FmView& f = A.fm[o];
                    idx_t rl[4] = {0, 0, 0, 0}, ru[4] = {0, 0, 0, 0};
                    if (ext || ends) {
                        rank_all(f, cl, rl);
                        rank_all(f, cu + 1, ru);
                        probes += 2;
                    }
                    if (ends) {
                        const idx_t ea = f.Cf[0] + (cl - (rl[0] + rl[1] + rl[2] + rl[3]));
                        const idx_t eb2 = f.Cf[0] + ((cu + 1) - (ru[0] + ru[1] + ru[2] + ru[3])) - 1;
                        if (ea <= eb2) {
                            const size_t me = mbase_w + size_t(j) * PMAX + i;
                            S.em_l[me] = ea;
                            S.em_u[me] = eb2;
                            atomicMin(&sm.hit[j], i);
                        }
                    }
                    if (ext) {
                        #pragma unroll
                        for (int a = 1; a <= 4; ++a) {
                            const int ch = o == 0 ? complement(a) : a;
                            const idx_t lo = f.Cf[ch] + pick4(rl, ch);
                            const idx_t hi = f.Cf[ch] + pick4(ru, ch) - 1;
                            if (lo <= hi) {
                                const size_t x = xbase_w + (size_t(j) * 4 + (a - 1)) * PMAX + i;
                                S.x_ll[x] = lo;
                                S.x_uu[x] = hi;
                                S.x_meta[x] = m;
                                atomicOr(&sm.mask[j][a - 1][i >> 6], 1ull << (i & 63));
                                atomicMax(&sm.cml[j][a - 1], meta_len(m));
                                atomicAdd(&sm.ctr[j][a - 1], unsigned(hi - lo + 1));
                            }
                        }
                    }
                }
                }
                __syncwarp();
                // (3) own control: emit, or record the four sets
                bool place = false;
                if (go) {
                    const int h = sm.hit[lane];
                    bool popped = false;
                    if (h != 0x7fffffff) {
                        const size_t me = mbase_w + size_t(lane) * PMAX + h;
                        const idx_t lll = S.em_l[me], uuu = S.em_u[me];
                        const uint32_t hm = S.t_meta[tb + F.pos + h];
                        const idx_t endk = uuu + 1;      // k < uuu + 1: no iteration when uuu + 1 wraps
                        const idx_t cnt = endk > lll ? endk - lll : 0;
                        const idx_t* rix = A.fm[cand_index(meta_type(hm))].reads_index;
                        if (cnt > 0) probes.add(0, sectors_of(rix + lll, size_t(cnt) * sizeof(idx_t)));
                        for (idx_t k = 0; k < cnt; ++k) {
                            const idx_t rr = __ldg(rix + (lll + k));
                            if (rr == self) continue;
                            if (sc + 1 > 65535) { status = ERR_TOO_MANY; break; }
                            if (ne + 1 > S.ebcap) { status = OVF_EDGES; break; }
                            S.e_dest[eb + ne] = rr;
                            S.e_trans[eb + ne] = F.trans;
                            S.e_meta[eb + ne] = hm;
                            ++ne;
                            ++sc;
                        }
                        if (status != OVF_NONE) {
                            active = false;
                        } else if (cnt > 0) {           // flag: this branch is finished
                            popped = true;
                            entering = false;
                            if (sp == 0) active = false;
                            else {
                                F = fr[--sp];
                                level = F.level;
                            }
                        }
                    }
                    if (!popped && active) {
                        int c[4];
                        int run = 0;
                        #pragma unroll
                        for (int a = 0; a < 4; ++a) {
                            c[a] = broad ? popc_words<MW>(sm.mask[lane][a]) : int((sm.cnt[lane] >> (8 * a)) & 0xffu);
                            sm.setoff[lane][a] = run;
                            run += c[a];
                        }
                        if (int(F.free) + run > CAP) {
                            status = OVF_STACK;
                            active = false;
                        } else {
                            F.cbase = F.free;
                            F.csz4 = uint64_t(c[0]) | (uint64_t(c[1]) << 16) | (uint64_t(c[2]) << 32) |
                                     (uint64_t(c[3]) << 48);
                            F.cml4 = uint64_t(sm.cml[lane][0]) | (uint64_t(sm.cml[lane][1]) << 16) |
                                     (uint64_t(sm.cml[lane][2]) << 32) | (uint64_t(sm.cml[lane][3]) << 48);
                            F.ctr[0] = int32_t(sm.ctr[lane][0]);
                            F.ctr[1] = int32_t(sm.ctr[lane][1]);
                            F.ctr[2] = int32_t(sm.ctr[lane][2]);
                            F.ctr[3] = int32_t(sm.ctr[lane][3]);
                            F.next_a = 1;
                            entering = false;
                            place = broad;
                        }
                    }
                }
                if (any_broad) {
                // (4) pack the sets of every larger task into its stack, in entry order
                sm.cbase[lane] = F.cbase;
                const int totx = warp_prefix(place ? 4 * int(F.size) : 0, sm.pref);
                __syncwarp();
                for (int e = lane; e < totx; e += 32) {
                    const int j = owner_of(sm.pref, e);
                    const int rel = e - sm.pref[j];
                    const int Pj = (sm.pref[j + 1] - sm.pref[j]) >> 2;
                    const int a = rel / Pj, i = rel - a * Pj;
                    const unsigned long long* mk = sm.mask[j][a];
                    if ((mk[i >> 6] >> (i & 63)) & 1) {
                        const int dst = int(sm.cbase[j]) + sm.setoff[j][a] + popc_below<MW>(mk, i);
                        const size_t x = xbase_w + (size_t(j) * 4 + a) * PMAX + i;
                        const size_t t = tbase_w + size_t(j) * CAP + dst;
                        S.t_ll[t] = S.x_ll[x];
                        S.t_uu[t] = S.x_uu[x];
                        S.t_meta[t] = S.x_meta[x];
                    }
                }
                }
                __syncwarp();
            }
        }
        }
        if (!Q.count) break;
    }
    if (Q.count == 0 || cur >= 0) add_probes(O, probes);
}

// ------------------------------------------------------------------------------ lean tier
//
// A warp takes 32 reads.  The rows to check of each read's two chains of a side are found lane by
// lane (k-mer table, narrow_rows); then the rows of all 32 reads are taken one a lane, so that 32
// suffix-array entries are in flight at once whatever the reads' own numbers of rows.  Rows at an offset that can be a candidate wait in a queue until a warp's worth is there
// to compare its texts, and a row that is a candidate takes the next slot of its read.  Each lane
// then reduces its read by sorted continuations.  A read the scan does not serve or with more than
// kRedMax candidates on a side is listed for the block tier: the fast tier's walk and DFS in between
// was slower for every kind of such reads, whether it could hold them or not (1.5 M bases of 100-base
// reads with 2 % dinucleotide runs, 2,165 such reads, 431 of which it could: 36 ms with it, 1.6
// without; with half the genome in repeats, 565 and 555: 3.4 and 1.9; 400x coverage, 38 thousand and
// 6 thousand: 8.6 and 5.3) but one: where depth-t intervals are large by chance (lean_misses_by_chance).
//
// Bound by DRAM at random sectors (4.1 TB/s, of which every second sector of a 64-byte fetch goes
// unused): k-mer table, kx, suffix array, text.  5.4 M reads of 100 bases, 566 M suffixes, 64-bit
// index: 7.3 ms, against 13.5 with one thread per read throughout (10 of 32 lanes active) and I_t
// found by bisection; 1.2 M reads, 123 M suffixes: 1.5 against 2.4.  Eight CTAs of 64 registers per
// SM; six or ten were 3 to 10 % slower.
constexpr int kLeanThreads = 128;

template <int W>
__global__ void __launch_bounds__(kLeanThreads, 8) k_search_lean(SearchArgs A0, SearchOut O0, WarpScratch S,
                                                                SearchQueue Q, int per) {
    __shared__ SearchBatch s_b[kLeanThreads / 32];
    __shared__ int s_pref[kLeanThreads / 32][33], s_m[kLeanThreads / 32][32];
    __shared__ idx_t s_qid[kLeanThreads / 32][64];              // rows waiting for their text to be checked:
    __shared__ uint32_t s_qo[kLeanThreads / 32][64];            // read, and offset | lane << 16 | chain << 21
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const size_t gw = size_t(blockIdx.x) * (kLeanThreads / 32) + wid;
    const size_t nw = size_t(gridDim.x) * (kLeanThreads / 32);
    SearchBatch& B = s_b[wid];
    const SearchArgs& A = B.a;
    const SearchOut& O = B.o;
    int* const pref = s_pref[wid];
    int* const slots = s_m[wid];
    idx_t* const qid = s_qid[wid];
    uint32_t* const qo = s_qo[wid];
    if (Q.count == 0) {
        if (lane == 0) {
            B.a = A0;
            B.o = O0;
        }
        __syncwarp();
    }
    const size_t ebase = gw * 32 * size_t(S.ebcap) + lane;      // edge i of a lane at ebase + 32 i
    const size_t rbase = gw * 32 * size_t(kRedMax);
    Tally probes;
    int cur = -1;
    for (size_t iter = 0;; ++iter) {
        size_t group, gend;
        if (Q.count) {
            unsigned it = 0;
            if (lane == 0) it = atomicAdd(Q.next, 1u);
            it = __shfl_sync(0xffffffffu, it, 0);
            if (it >= Q.count) break;
            const int b = int(Q.item_batch[it]);
            group = Q.item_group[it];
            gend = group + Q.groups_per_item;
            if (b != cur) {
                if (cur >= 0) add_probes(O, probes);
                probes = Tally{};
                __syncwarp();
                load_batch(B, Q.batches + b, lane);
                cur = b;
            }
        } else {
            group = gw + iter * nw;
            gend = group + 1;
            if (group * per >= size_t(A.num_reads)) break;
        }
        for (; group < gend && group * per < size_t(A.num_reads); ++group) {
            const int L = A.L, t = A.t, M = L - t;
            const size_t r = group * per + lane;
            const idx_t self = idx_t(r);
            const bool have = lane < per && r < size_t(A.num_reads);
            bool ok = have;
            int ne = 0, status = OVF_NONE;
            int count_b = 0, count_f = 0;
            int32_t olp_b = 0, olp_f = 0;
            // B side: B-F then B-B candidates, then extract_bw_edges (src/string_graph.c:824-825);
            // then the F side: F-B, F-F, extract_fw_edges (:828-829).  Both kinds of a side take
            // their pattern from the same text: the first as it is, the second its complement.
            #pragma unroll 1
            for (int side = 0; side < 2; ++side) {
                const int k0 = side ? PQ_FB : PQ_BF, k1 = side ? PQ_FF : PQ_BB;
                const FmView* f0 = A.fm + walked_index(k0);
                const FmView* f1 = A.fm + walked_index(k1);
                idx_t first[2] = {0, 0}, end[2] = {0, 0};
                uint64_t P0[kScanWords] = {}, P1[kScanWords] = {};
                if (ok) {
                    pattern_words(A.fm, L, t, k0, self, P0, probes);
                    #pragma unroll
                    for (int w = 0; w < kScanWords; ++w) P1[w] = ~P0[w];
                }
                if (A.sa_seed == 2) {
                    if (ok) ok = learned_rows(A, f0, f1, P0, P1, first, end, probes);
                    __syncwarp();
                } else {
                    const int k = A.seed_k;
                    if (ok) {
                        kmer_rows(*f0, uint32_t(P0[0] >> (64 - 2 * k)), first[0], end[0]);
                        kmer_rows(*f1, uint32_t(P1[0] >> (64 - 2 * k)), first[1], end[1]);
                        probes.add(2, 2);
                        #pragma unroll
                        for (int q = 0; q < 2; ++q) end[q] = end[q] < first[q] ? first[q] : end[q] + 1;
                    }
                    narrow_rows(*f0, k, t, P0[0], first[0], end[0], probes);
                    narrow_rows(*f1, k, t, P1[0], first[1], end[1], probes);
                    const int bare = per < 32 || L <= 64 || t == k ? kScanDirect : kScanBare;
                    if (ok && (end[0] - first[0] > idx_t(f0->kx_bases ? kScanDirect : bare) ||
                               end[1] - first[1] > idx_t(f1->kx_bases ? kScanDirect : bare))) {
                        const idx_t lo[2] = {first[0], first[1]}, hi[2] = {end[0], end[1]};
                        sa_bounds2(f0, f1, A.dl, P0, P1, t < 32 * kScanWords ? t : 32 * kScanWords, lo, hi, first, end, probes);
                        ok = end[0] - first[0] <= idx_t(kScanMax) && end[1] - first[1] <= idx_t(kScanMax);
                    }
                }
                slots[lane] = 0;
                __syncwarp();
                // a row that passed the offset test: its read against the whole pattern, and its
                // continuation (M - o bases of the walked text after the pattern) if it matches
                const uint64_t* const pks = f0->pk;             // both patterns' source
                auto check = [&](int i, unsigned lanes) {
                    const idx_t rp = qid[i];
                    const uint32_t v = qo[i];
                    const int o = int(v & 0xffffu), j = int((v >> 16) & 31u), d = t + o, len = M - o;
                    const bool cmpl = (v >> 21) != 0;
                    const FmView& fa = cmpl ? *f1 : *f0;
                    const size_t text = size_t(rp) * size_t(L);
                    const size_t src = (group * per + size_t(j)) * size_t(L) + size_t(len);
                    probes.add(0, base_sectors(text, d));
                    if (!text_matches(fa.pk, text, pks, src, d, cmpl, lanes)) return;
                    const int slot = atomicAdd(&slots[j], 1);
                    if (slot >= kRedMax) return;
                    const size_t pos = text + size_t(d), at = rbase + size_t(slot) * kRedStride + size_t(j);
                    const uint32_t flip = walked_index(cmpl ? k1 : k0) ? ~0u : 0u;
                    const uint64_t* w = fa.pk + (pos >> 5);
                    const int s = int(pos & 31);
                    uint64_t a0 = __ldg(w);
                    #pragma unroll
                    for (int q = 0; q < W; ++q) {
                        const int left = len - 32 * q;
                        if (left <= 0) break;
                        const uint64_t a1 = __ldg(w + q + 1);
                        uint32_t h, l;
                        shift_bases(a0, a1, s, h, l);
                        S.r_k[q * S.r_plane + at] = (uint64_t((h ^ flip) & half_mask(left, 0)) << 32) |
                                                    ((l ^ flip) & half_mask(left, 1));
                        a0 = a1;
                    }
                    probes.add(0, base_sectors(pos, len));
                    S.r_id[at] = rp;
                    S.r_meta[at] = pack_meta(d, cmpl ? k1 : k0);
                };
                int waiting = 0;
                #pragma unroll 1
                for (int q = 0; q < 2; ++q) {
                    const idx_t* const sa = q ? f1->sa : f0->sa;
                    const idx_t mine = q ? first[1] : first[0];
                    const int total = warp_prefix(ok ? int((q ? end[1] : end[0]) - mine) : 0, pref);
                    for (int e0 = 0; e0 < total; e0 += 32) {
                        const int e = e0 + lane;
                        const int j = owner_of(pref, e < total ? e : total - 1);
                        const idx_t row = __shfl_sync(0xffffffffu, mine, j) + idx_t(e - pref[j]);
                        int o = M;
                        idx_t rp = 0;
                        if (e < total) {
                            const idx_t p = __ldg(sa + row);
                            rp = read_of(p, A.dl);
                            o = int(p - rp * idx_t(L));
                            probes.add(2, 1);
                        }
                        const unsigned pass = __ballot_sync(0xffffffffu, o < M);
                        if (o < M) {
                            const int i = waiting + __popc(pass & ((1u << lane) - 1u));
                            qid[i] = rp;
                            qo[i] = uint32_t(o) | (uint32_t(j) << 16) | (uint32_t(q) << 21);
                        }
                        __syncwarp();
                        waiting += __popc(pass);
                        if (waiting >= 32) {                    // a full warp's worth
                            waiting -= 32;
                            check(waiting + lane, 0xffffffffu);
                            __syncwarp();
                        }
                    }
                    __syncwarp();
                }
                if (lane < waiting) check(lane, (1u << waiting) - 1u);
                __syncwarp();
                const int m = slots[lane];
                if (m > kRedMax) {
                    ok = false;
                    status = OVF_STACK;
                }
                int count = 0;
                if (ok && m && status == OVF_NONE)
                    status = reduce_gathered<W>(L, S, self, side, rbase + lane, m, ebase, 32, ne, count);
                if (side == 0) {
                    olp_b = m;
                    count_b = count;
                } else {
                    olp_f = m;
                    count_f = count;
                }
                __syncwarp();
            }
            if (have && (!ok || status != OVF_NONE)) {   // the fast or the block tier redoes this read
                if (ok) O.status[r] = uint8_t(status);
                if (!ok && status == OVF_NONE && A.miss_list) A.miss_list[atomicAdd(A.miss_count, 1u)] = self;
                else O.ovf_list[atomicAdd(O.ovf_count, 1u)] = self;
            }
            // one reservation of edge slots for the warp's reads
            const int mine = have && ok && status == OVF_NONE ? ne : 0;
            const int edges = warp_prefix(mine, pref);
            unsigned long long base = 0;
            if (lane == 0 && edges) base = atomicAdd(O.e_count, (unsigned long long)edges);
            base = __shfl_sync(0xffffffffu, base, 0) + (unsigned long long)pref[lane];
            __syncwarp();
            if (!have || !ok || status != OVF_NONE) continue;
            if (ne && base + ne > O.e_cap) {
                O.status[r] = OVF_POOL;
                const unsigned k = atomicAdd(O.ovf_count, 1u);
                O.ovf_list[k] = self;
                continue;
            }
            for (int e = 0; e < ne; ++e) {
                const size_t q = ebase + size_t(e) * 32;
                const uint32_t mt = S.e_meta[q];
                O.e_dest[base + e] = S.e_dest[q];
                O.e_trans[base + e] = S.e_trans[q];
                O.e_len[base + e] = uint16_t(meta_len(mt));
                O.e_type[base + e] = uint8_t(meta_type(mt));
            }
            O.status[r] = OVF_NONE;
            O.num_B[r] = uint16_t(count_b);
            O.num_F[r] = uint16_t(count_f);
            O.olp_B[r] = olp_b;
            O.olp_F[r] = olp_f;
            O.edge_src[r] = base;
        }
        __syncwarp();
    }
    if (Q.count == 0 || cur >= 0) add_probes(O, probes);
}

// Reads the scan does not serve have a depth-t interval of more than kScanMax rows.  With long overlaps
// those are repeats and low complexity, whose walks and DFS are long: the block tier's.  With short ones
// an ordinary read's interval is that large by chance, rows / 4^t (several times that where bases are
// skewed).  Such a read has few candidates: the fast tier, 32 reads a warp, takes 25 ns a read, the
// block tier, a CTA a read, 90.  But its slowest warp takes 0.8 ms, which 9 thousand reads of the block
// tier do not: kFastMisses.  Whole searches in ms, misses to the fast tier (and on where a side has more than
// kRedMax candidates) and to the block tier, reads of 100 bases at 20x, GC 41 %:
//   rows 54 M, t = 10 (51 rows by chance, 5 thousand misses): 6.1 and 5.4;  78 M (74, 46 thousand): 9.6 and 12.1;
//   108 M (103, 198 thousand): 17.0 and 29.8;  431 M (411, 4.2 M): 210 and 415;  861 M, t = 11, 64-bit (205, 6.1
//   M): 267 and 699;  t = 10 (821, 8.6 M, of which 3.1 M go on): 952 and 1006.
bool lean_misses_by_chance(size_t rows, int t) { return t < 32 && (rows >> (2 * t)) >= size_t(kScanMax) / 8; }

int search_lean_blocks(int L, int M, int num_sms) {
    (void)L;
    int per_sm = 0;
    const cudaError_t e = lam_words(M) == 2
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search_lean<2>, kLeanThreads, 0)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search_lean<kLamWords>, kLeanThreads, 0);
    if (e != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    return per_sm * num_sms;
}

int search_fast_blocks(int L, int M, int num_sms) {
    const int words = (L + 15) / 16;
    const size_t smem = size_t(words) * 32 * kWarpsPerCta * sizeof(uint32_t);
    int per_sm = 0;
    const cudaError_t e = lam_words(M) == 2
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search_fast<2, kTaskCap, kTaskFrames, kPMax>, 32 * kWarpsPerCta, smem)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_search_fast<kLamWords, kTaskCap, kTaskFrames, kPMax>, 32 * kWarpsPerCta, smem);
    if (e != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return per_sm * num_sms;
}

static size_t scratch_layout(int M_max, size_t nwarps, int ebcap, void* base, WarpScratch* S, int cap = kTaskCap,
                             int frames = kTaskFrames, int pmax = kPMax, bool lean = false) {
    const size_t M = size_t(M_max), pool = std::max(size_t(kFastPool), 4 * M), edg = nwarps * 32 * size_t(ebcap);
    const size_t dfs = lean ? 0 : nwarps;                   // warps that walk and run the DFS
    const size_t cand = dfs * 32 * 4 * M, tsk = dfs * 32 * size_t(cap), spr = dfs * 32 * 4 * size_t(pmax);
    const size_t emb = dfs * 32 * size_t(pmax), frm = dfs * 32 * size_t(frames);
    char* p = static_cast<char*>(base);
    size_t used = 0;
    auto take = [&](size_t bytes) {
        char* q = p ? p + used : nullptr;
        used += (bytes + 255) & ~size_t(255);
        return q;
    };
    WarpScratch T{};
    T.c_ll = reinterpret_cast<idx_t*>(take(cand * sizeof(idx_t)));
    T.c_uu = reinterpret_cast<idx_t*>(take(cand * sizeof(idx_t)));
    T.c_meta = reinterpret_cast<uint32_t*>(take(cand * 4));
    T.p_ll = reinterpret_cast<idx_t*>(take(dfs * pool * sizeof(idx_t)));
    T.p_uu = reinterpret_cast<idx_t*>(take(dfs * pool * sizeof(idx_t)));
    T.p_meta = reinterpret_cast<uint32_t*>(take(dfs * pool * 4));
    T.queue = reinterpret_cast<FastTask*>(take(dfs * kFastQueue * sizeof(FastTask)));
    T.pool = int(pool);
    T.e_dest = reinterpret_cast<idx_t*>(take(edg * sizeof(idx_t)));
    T.e_trans = reinterpret_cast<int32_t*>(take(edg * 4));
    T.e_meta = reinterpret_cast<uint32_t*>(take(edg * 4));
    T.t_ll = reinterpret_cast<idx_t*>(take(tsk * sizeof(idx_t)));
    T.t_uu = reinterpret_cast<idx_t*>(take(tsk * sizeof(idx_t)));
    T.t_meta = reinterpret_cast<uint32_t*>(take(tsk * 4));
    T.x_ll = reinterpret_cast<idx_t*>(take(spr * sizeof(idx_t)));
    T.x_uu = reinterpret_cast<idx_t*>(take(spr * sizeof(idx_t)));
    T.x_meta = reinterpret_cast<uint32_t*>(take(spr * 4));
    T.em_l = reinterpret_cast<idx_t*>(take(emb * sizeof(idx_t)));
    T.em_u = reinterpret_cast<idx_t*>(take(emb * sizeof(idx_t)));
    T.frames = reinterpret_cast<TFrame*>(take(frm * sizeof(TFrame)));
    const size_t red = nwarps * 32 * size_t(kRedMax);
    T.r_k = reinterpret_cast<uint64_t*>(take(red * 8 * kLamWords));
    T.r_plane = red;
    T.r_id = reinterpret_cast<idx_t*>(take(red * sizeof(idx_t)));
    T.r_meta = reinterpret_cast<uint32_t*>(take(red * 4));
    T.r_emit = reinterpret_cast<uint32_t*>(take(red * 4));
    T.ebcap = ebcap;
    T.mstride = int(M);
    if (S) *S = T;
    return used;
}

static size_t lean_layout(int M_max, size_t nwarps, int ebcap, void* base, WarpScratch* S) {
    return scratch_layout(M_max, nwarps, ebcap, base, S, kTaskCap, kTaskFrames, kPMax, true);
}

size_t warp_scratch_bytes(int L, int t, size_t nwarps, int ebcap) {
    return scratch_layout(L - t, nwarps, ebcap, nullptr, nullptr);
}

cudaError_t search_fast(const SearchArgs& a, const SearchOut& o, int blocks, void* scratch, size_t scratch_bytes,
                        int ebcap, cudaStream_t st, const idx_t* list, const unsigned* count) {
    const size_t nwarps = size_t(blocks) * kWarpsPerCta;
    WarpScratch S;
    if (scratch_bytes < scratch_layout(a.L - a.t, nwarps, ebcap, scratch, &S)) return cudaErrorInvalidValue;
    const int words = (a.L + 15) / 16;
    size_t smem = size_t(words) * 32 * kWarpsPerCta * sizeof(uint32_t);
    SearchQueue Q{};
    Q.read_list = list;
    Q.list_count = count;
    Q.per = 32;
    Q.dfs_max = list ? 0 : kTaskCap;        // of listed reads (the lean tier's misses) the sorted reduction only
    if (lam_words(a.L - a.t) == 2) k_search_fast<2, kTaskCap, kTaskFrames, kPMax><<<blocks, 32 * kWarpsPerCta, smem, st>>>(a, o, S, Q);
    else k_search_fast<kLamWords, kTaskCap, kTaskFrames, kPMax><<<blocks, 32 * kWarpsPerCta, smem, st>>>(a, o, S, Q);
    note_launch();
    return cudaGetLastError();
}

// Reads a warp takes: 32, or 16, 8 or 4 where there are not 32 for every warp resident.  A warp takes the
// rows of its reads 32 at a time, so a quarter of the reads is nearly a quarter of its time (4.9
// thousand reads of 100 bases: 87 us with 32 a warp, 31 with 4).
static int lean_reads(size_t num_reads, int blocks) {
    int per = 32;
    while (per > 4 && num_reads <= size_t(blocks) * (kLeanThreads / 32) * size_t(per / 2)) per /= 2;
    return per;
}

cudaError_t search_lean(const SearchArgs& a, const SearchOut& o, int blocks, void* scratch, size_t scratch_bytes, int ebcap,
                        cudaStream_t st) {
    WarpScratch S;
    if (scratch_bytes < lean_layout(a.L - a.t, size_t(blocks) * (kLeanThreads / 32), ebcap, scratch, &S))
        return cudaErrorInvalidValue;
    SearchQueue none{};
    const int per = lean_reads(size_t(a.num_reads), blocks);
    if (lam_words(a.L - a.t) == 2) k_search_lean<2><<<blocks, kLeanThreads, 0, st>>>(a, o, S, none, per);
    else k_search_lean<kLamWords><<<blocks, kLeanThreads, 0, st>>>(a, o, S, none, per);
    note_launch();
    return cudaGetLastError();
}

// Queued lean search: one persistent lean launch over the queue (kernel built for the words of
// M_max; no host sync).
cudaError_t search_lean_queue(const SearchQueue& q, int M_max, int blocks, void* scratch, size_t scratch_bytes, int ebcap,
                              cudaStream_t st) {
    WarpScratch S;
    if (scratch_bytes < lean_layout(M_max, size_t(blocks) * (kLeanThreads / 32), ebcap, scratch, &S)) return cudaErrorInvalidValue;
    SearchArgs a0{};
    SearchOut o0{};
    if (lam_words(M_max) == 2) k_search_lean<2><<<blocks, kLeanThreads, 0, st>>>(a0, o0, S, q, 32);
    else k_search_lean<kLamWords><<<blocks, kLeanThreads, 0, st>>>(a0, o0, S, q, 32);
    note_launch();
    return cudaGetLastError();
}

size_t lean_scratch_bytes(int L, int t, int blocks, int ebcap) {
    return lean_layout(L - t, size_t(blocks) * (kLeanThreads / 32), ebcap, nullptr, nullptr);
}

// ------------------------------------------------------------------------------ block tier
//
// Reads the lean tier hands over are mostly the ones with many candidates -- low-complexity sequence,
// where a read's side can have thousands.  One thread per (read, side) walks the chains of all of
// them first (k_block_walk: chain_pair, from exact k-mer seeds, with the reference's depths), so
// that the dependent steps of thousands of walks overlap.  Then one CTA takes each read: every
// candidate group is expanded into its candidates (read id from the suffix array, continuation from
// the packed text) and each side is reduced in shared memory by sorting (k_search_block).  A side
// with more candidates than the larger of its two sizes goes to the variant with everything in
// global memory (k_search_block_global), and only one beyond that variant's capacity to the heavy
// and wide tiers.

// The candidate groups of one (read, side): n[q] of kind q at grp[q * M ..], their candidates' number
// (0xffffffff: more than any block kernel holds) and the overlaps counted.
struct BlockSide {
    int n[2];
    int32_t olp;
    unsigned m;
};
constexpr int kWalkThreads = 64;

__global__ void __launch_bounds__(kWalkThreads) k_block_walk(SearchArgs A, SearchOut O, const idx_t* list, unsigned count,
                                                             Cand* groups, BlockSide* sides) {
    extern __shared__ uint32_t s_reads[];
    const unsigned i = (blockIdx.x * kWalkThreads + threadIdx.x);
    Tally probes;
    if (i < 2 * count) {
        const int side = int(i & 1u), M = A.L - A.t;
        load_read(A, list[i >> 1], s_reads + threadIdx.x, kWalkThreads, probes);
        const ReadView rd{s_reads + threadIdx.x, kWalkThreads};
        Cand* g = groups + size_t(i) * size_t(2 * M);
        BlockSide b{};
        chain_pair(A, A.fm, rd, side ? PQ_FB : PQ_BF, side ? PQ_FF : PQ_BB, b.n, b.olp, probes, SlotsStack{g, M});
        unsigned long long m = 0;               // group sizes are index-wide: summed in 64 bits, stopped past 2^31
        for (int q = 0; q < 2; ++q)
            for (int j = 0; j < b.n[q] && m < (1ull << 31); ++j) {
                const Cand& c = g[q * M + j];
                m += (unsigned long long)(c.uu - c.ll) + 1ull;
            }
        b.m = m < (1ull << 31) ? unsigned(m) : 0xffffffffu;
        sides[i] = b;
    }
    add_probes(O, probes);
}

// What k_search_block keeps per candidate in its CTA's region of global memory (L2-resident), each
// an array of CAP: continuation words, read id, (overlap, kind) and, of either side, the emitted
// edges.
__host__ __device__ constexpr size_t block_region_bytes(int cap, int nw) {
    return size_t(cap) * (size_t(nw) * 8 + sizeof(idx_t) + 4 + 2 * (sizeof(idx_t) + 4 + 4));
}
// and in shared memory: the sort key (the walk's record after the sort), the order, and the group
// prefix sums
constexpr size_t block_smem_bytes(int cap) { return size_t(cap) * 10 + (2 * 256 + 1 + 31) * 4; }
constexpr int kBlockSmall = 4096, kBlockMid = 8192, kBlockLarge = 16384;    // candidates a side, by 256, 512 and 512 threads

// One read a CTA.  Each side's candidates are ordered by (continuation words, zero past the end;
// length; read id) with a bitonic sort in shared memory.  In low-complexity sequence most
// continuations start with the same long run, so a key of their first words would seldom tell them
// apart: the key is relative to one of them, the pivot p.  With l the common prefix of a continuation
// and p, its highest 10 bits are l where the continuation ends there or is smaller than p, 1023 - l
// where it is larger, and the next 53 the 26 1/2 bases from l on: continuations of one side and one l
// share their first l bases, and of two that leave p at different places the one that leaves it later
// is nearer to p.  (One that ends at l is a prefix of every other that shares more than l bases with p
// and sorts before it: its padding is the smallest base.)  The lowest bit is clear in a prefix of
// p, which sorts before what goes on with the smallest base; equal keys without it are equal strings,
// other equal keys are compared by all words.
//
// In that order a continuation is followed by its extensions: its class, found for all places at once
// by a prefix scan (below).  The candidates equal to their class's shortest are emitted, in DFS order.
//
// Bound by the sort's instructions and its barriers.  The 3,645 run reads of the 200 Mbp workload at
// 1/100 genome (150 bases, up to 6.7 thousand candidates of a kind) took 58 ms by pair tests in shared
// memory and radix passes in global memory; 19 with the first words as keys; 16 with keys relative to
// a pivot and one warp walking from class to class; 6 with the classes found by the scan, 5.2 with
// equal keys compared only from where they may differ.  (Two steps of the network at a time gave 5.0.)
template <int CAP, int T>
__global__ void __launch_bounds__(T) k_search_block(SearchArgs A, SearchOut O, const idx_t* list, unsigned count, const Cand* groups,
                                                    const BlockSide* sides, unsigned* next, unsigned char* region,
                                                    unsigned lowest, unsigned highest, idx_t* next_list, unsigned* next_count) {
    extern __shared__ __align__(16) unsigned char smem_dyn[];
    uint64_t* const key = reinterpret_cast<uint64_t*>(smem_dyn);
    uint16_t* const ord = reinterpret_cast<uint16_t*>(key + CAP);
    unsigned* const pref = reinterpret_cast<unsigned*>(ord + CAP);
    __shared__ unsigned s_item, s_sum[T / 32];
    __shared__ int s_ne[2], s_pivot;
    __shared__ unsigned long long s_base;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    constexpr int NW = T / 32;
    const int L = A.L, M = L - A.t, nw = (M + 31) / 32;
    unsigned char* at = region + size_t(blockIdx.x) * block_region_bytes(CAP, nw);
    uint64_t* const cw = reinterpret_cast<uint64_t*>(at); at += size_t(CAP) * nw * 8;
    idx_t* const cid = reinterpret_cast<idx_t*>(at); at += size_t(CAP) * sizeof(idx_t);
    idx_t* const e_id = reinterpret_cast<idx_t*>(at); at += size_t(2 * CAP) * sizeof(idx_t);
    uint32_t* const cmeta = reinterpret_cast<uint32_t*>(at); at += size_t(CAP) * 4;
    uint32_t* const e_meta = reinterpret_cast<uint32_t*>(at); at += size_t(2 * CAP) * 4;
    int32_t* const e_trans = reinterpret_cast<int32_t*>(at);
    Tally probes;
    while (true) {
        if (tid == 0) s_item = atomicAdd(next, 1u);
        __syncthreads();
        const unsigned item = s_item;
        if (item >= count) break;
        const BlockSide sb[2] = {sides[2 * item], sides[2 * item + 1]};
        const unsigned most = max(sb[0].olp ? sb[0].m : 0u, sb[1].olp ? sb[1].m : 0u);
        __syncthreads();
        if (most < lowest || most > highest) continue;          // the other size's, or the next tier's
        const idx_t self = list[item];
        if (tid < 2) s_ne[tid] = 0;
        for (int side = 0; side < 2; ++side) {
            if (sb[side].olp == 0) continue;                    // src/string_graph.c:824, 828
            const int n0 = sb[side].n[0], ng = n0 + sb[side].n[1], m = int(sb[side].m);
            const Cand* g = groups + (size_t(2 * item) + side) * size_t(2 * M);
            // exclusive prefix of the group sizes, two groups a thread (ng <= 2 M <= 512)
            {
                unsigned v[2] = {0, 0};
                #pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int i = 2 * tid + q;
                    if (i < ng) {
                        const Cand& c = g[i < n0 ? i : M + (i - n0)];
                        v[q] = unsigned(c.uu - c.ll) + 1u;
                    }
                }
                unsigned x = v[0] + v[1];
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == 31) s_sum[wid] = x;
                __syncthreads();
                unsigned run = x - v[0] - v[1];
                for (int w = 0; w < wid; ++w) run += s_sum[w];
                if (2 * tid <= ng) pref[2 * tid] = run;
                if (2 * tid + 1 <= ng) pref[2 * tid + 1] = run + v[0];
                __syncthreads();
            }
            // every candidate's read id and continuation
            for (int i = tid; i < m; i += T) {
                int lo = 0, hi = ng - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (pref[mid] <= unsigned(i)) lo = mid;
                    else hi = mid - 1;
                }
                const Cand& c = g[lo < n0 ? lo : M + (lo - n0)];
                const idx_t row = c.ll + idx_t(unsigned(i) - pref[lo]);
                const int type = int(c.type), d = int(c.len);
                const idx_t rp = read_of(__ldg(A.fm[cand_index(type)].sa + row), A.dl);
                for (int w = 0; w < nw; ++w) {
                    const uint64_t x = 32 * w < L - d ? continuation_word(A, type, rp, d, w) : 0;
                    cw[size_t(w) * CAP + i] = x;
                }
                probes.add(2, 1 + base_sectors(size_t(rp) * L + size_t(d), L - d));
                cid[i] = rp;
                cmeta[i] = pack_meta(d, type);
                ord[i] = uint16_t(i);
            }
            __syncthreads();
            auto length = [&](int i) { return L - meta_len(cmeta[i]); };
            // common prefix of candidates i and j
            auto shared_prefix = [&](int i, int j) {
                const int n = min(length(i), length(j));
                for (int w = 0; 32 * w < n; ++w) {
                    const uint64_t z = cw[size_t(w) * CAP + i] ^ cw[size_t(w) * CAP + j];
                    if (z) return min(n, 32 * w + (__clzll((long long)z) >> 1));
                }
                return n;
            };
            // the pivot: of 32 candidates, the one that shares most with 8 of them
            if (wid == 0) {
                const int mine = int((unsigned long long)lane * unsigned(m) >> 5);
                unsigned sum = 0;
                for (int j = 2; j < 32; j += 4) sum += unsigned(shared_prefix(mine, int((unsigned long long)j * unsigned(m) >> 5)));
                const unsigned best = __reduce_max_sync(0xffffffffu, (sum << 5) | unsigned(lane));
                if (lane == 0) s_pivot = int((unsigned long long)(best & 31u) * unsigned(m) >> 5);
            }
            __syncthreads();
            const int pivot = s_pivot, lp = length(pivot);
            for (int i = tid; i < m; i += T) {
                const int n = length(i), l = shared_prefix(i, pivot);
                const int w = l >> 5, sh = 2 * (l & 31);
                const uint64_t x0 = w < nw ? cw[size_t(w) * CAP + i] : 0;
                const uint64_t x1 = w + 1 < nw ? cw[size_t(w + 1) * CAP + i] : 0;
                const uint64_t rest = sh ? (x0 << sh) | (x1 >> (64 - sh)) : x0;     // zero past the end
                bool larger = false;
                if (l < n) larger = l == lp || rest >> 62 > ((cw[size_t(w) * CAP + pivot] << sh) >> 62);
                key[i] = (uint64_t(unsigned(larger ? 1023 - l : l)) << 54) | ((rest >> 11) << 1) | uint64_t(l != n);
            }
            __syncthreads();
            // a before b, whose keys are equal.  Equal continuations of one kind stay as they were expanded,
            // in row order, which is ascending read id; of two kinds only one is emitted.
            auto before = [&](int a, int b, uint64_t k) {
                if (k & 1) {                // equal up to 26 bases past where both leave the pivot
                    const int l = int(k >> 54);
                    for (int w = ((l < 512 ? l : 1023 - l) + 26) >> 5; w < nw; ++w) {
                        const uint64_t x = cw[size_t(w) * CAP + a], y = cw[size_t(w) * CAP + b];
                        if (x != y) return x < y;
                    }
                    const int la = length(a), lb = length(b);
                    if (la != lb) return la < lb;
                }
                return a < b;
            };
            auto exchange = [&](int a, int b) {
                if (b >= m) return;
                const uint64_t x = key[a], y = key[b];
                if (x < y) return;
                const int p = ord[a], q = ord[b];
                if (x == y && before(p, q, x)) return;
                key[a] = y;
                key[b] = x;
                ord[a] = uint16_t(q);
                ord[b] = uint16_t(p);
            };
            for (int k = 2; k < 2 * m; k <<= 1) {
                const int half = k >> 1, pairs = (m + k - 1) / k * half;
                for (int i = tid; i < pairs; i += T) {          // the mirrored step: every comparator points up
                    const int q = i / half, o = i - q * half;
                    exchange(q * k + o, q * k + k - 1 - o);
                }
                __syncthreads();
                for (int j = half >> 1; j > 0; j >>= 1) {
                    for (int i = tid; i < pairs; i += T) {
                        const int a = ((i & ~(j - 1)) << 1) | (i & (j - 1));
                        exchange(a, a + j);
                    }
                    __syncthreads();
                }
            }
            // per place of the order, in the key's four 16-bit fields: common prefix with the place
            // before (later the class), length, flags, and (by class) the class's first place
            const int first_kind = side ? PQ_FB : PQ_BF;
            constexpr unsigned kSelf = 1, kFirst = 2, kEqual = 4, kFirstSame = 8;
            ushort4* const at4 = reinterpret_cast<ushort4*>(key);
            for (int k = tid; k < m; k += T) {
                const int c = ord[k];
                const int lcp = k > 0 ? shared_prefix(int(ord[k - 1]), c) : 0;
                at4[k] = make_ushort4(uint16_t(lcp), uint16_t(length(c)),
                                      uint16_t((cid[c] == self ? kSelf : 0u) | (meta_type(cmeta[c]) == first_kind ? kFirst : 0u)), 0);
            }
            // The shortest candidate that is a prefix of place k's, H(k) its length, starts k's class:
            // H(k) = H(k - 1) where that is at most k's common prefix with k - 1, else k's own length
            // (a longer prefix of k - 1 than H(k - 1) cannot reach k either).  Such steps compose,
            // (a1, b1) then (a2, b2) to (min(a1, a2), b1 <= a2 ? b1 : b2), so H is a prefix scan.
            const int rows = (m + 32 * NW - 1) / (32 * NW), k0 = wid * rows * 32;
            auto then = [](unsigned f, unsigned g) {            // a << 16 | b
                const unsigned a1 = f >> 16, b1 = f & 0xffffu, a2 = g >> 16, b2 = g & 0xffffu;
                return (min(a1, a2) << 16) | (b1 <= a2 ? b1 : b2);
            };
            auto step = [&](int k) {
                if (k >= m) return 0xffffffffu;                 // nothing
                const ushort4 v = at4[k];
                return (unsigned(v.x) << 16) | v.y;
            };
            __syncthreads();
            {
                unsigned f = 0xffffffffu;
                for (int q = 0; q < rows; ++q) {
                    unsigned x = step(k0 + 32 * q + lane);
                    #pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const unsigned y = __shfl_down_sync(0xffffffffu, x, o);
                        if (lane + o < 32) x = then(x, y);      // lane 0: the row's steps in order
                    }
                    f = then(f, __shfl_sync(0xffffffffu, x, 0));
                }
                if (lane == 0) s_sum[wid] = f;
            }
            __syncthreads();
            {
                unsigned f = 0xffffffffu;
                for (int w = 0; w < wid; ++w) f = then(f, s_sum[w]);
                int heads = 0;
                for (int q = 0; q < rows; ++q) {
                    const int k = k0 + 32 * q + lane;
                    unsigned x = step(k);
                    const unsigned lcp = x >> 16, len = x & 0xffffu;
                    #pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
                        if (lane >= o) x = then(y, x);
                    }
                    x = then(f, x);
                    const unsigned up = __shfl_up_sync(0xffffffffu, x, 1);
                    const bool head = k < m && ((lane ? up : f) & 0xffffu) > lcp;
                    const bool equal = k < m && len == (x & 0xffffu);
                    const unsigned hb = __ballot_sync(0xffffffffu, head);
                    if (k < m) {                                // class within the warp's places, for now
                        ushort4 v = at4[k];
                        v.x = uint16_t(heads + __popc(hb & (0xffffffffu >> (31 - lane))));
                        v.z = uint16_t(v.z | (equal ? kEqual : 0u) | (head ? 0x8000u : 0u));
                        at4[k] = v;
                    }
                    heads += __popc(hb);
                    f = __shfl_sync(0xffffffffu, x, 31);
                }
                __syncthreads();
                if (lane == 0) s_sum[wid] = unsigned(heads);
            }
            __syncthreads();
            int classes = 0;
            {
                int before_me = 0;
                for (int w = 0; w < NW; ++w) {
                    before_me += w < wid ? int(s_sum[w]) : 0;
                    classes += int(s_sum[w]);
                }
                for (int q = 0; q < rows; ++q) {
                    const int k = k0 + 32 * q + lane;
                    if (k >= m) break;
                    const int c = before_me + int(at4[k].x) - 1;
                    at4[k].x = uint16_t(c);
                    if (at4[k].z & 0x8000u) at4[c].w = uint16_t(k);
                }
            }
            __syncthreads();
            // a class with a first-kind candidate of exactly its continuation
            for (int k = tid; k < m; k += T) {
                const ushort4 v = at4[k];
                if ((v.z & (kEqual | kFirst)) == (kEqual | kFirst))
                    atomicOr(reinterpret_cast<unsigned*>(key + v.x) + 1, kFirstSame);
            }
            __syncthreads();
            auto emitted = [&](int k) {
                if (k >= m) return false;
                const ushort4 v = at4[k];
                return (v.z & kEqual) && !(v.z & kSelf) && ((v.z & kFirst) || !(at4[v.x].z & kFirstSame));
            };
            {
                int n = 0;
                for (int q = 0; q < rows; ++q) n += __popc(__ballot_sync(0xffffffffu, emitted(k0 + 32 * q + lane)));
                if (lane == 0) s_sum[wid] = unsigned(n);
            }
            __syncthreads();
            {
                const int ne0 = side ? s_ne[0] : 0;             // the F side's edges follow the B side's
                int ne = ne0, all = 0;
                for (int w = 0; w < NW; ++w) {
                    ne += w < wid ? int(s_sum[w]) : 0;
                    all += int(s_sum[w]);
                }
                for (int q = 0; q < rows; ++q) {
                    const int k = k0 + 32 * q + lane;
                    const bool em = emitted(k);
                    const unsigned e = __ballot_sync(0xffffffffu, em);
                    if (em) {
                        const int z = ne + __popc(e & ((1u << lane) - 1u)), c = ord[k], cls = at4[k].x;
                        e_id[z] = cid[c];
                        e_meta[z] = cmeta[c];
                        e_trans[z] = (cls + 1 < classes ? int(at4[cls + 1].w) : m) - int(at4[cls].w);
                    }
                    ne += __popc(e);
                }
                if (tid == 0) s_ne[side] = all;
            }
            __syncthreads();
        }
        __syncthreads();
        const int nb = s_ne[0], nf = s_ne[1], ne = nb + nf;
        if (tid == 0) {
            s_base = ne ? atomicAdd(O.e_count, (unsigned long long)ne) : 0ull;
            if (s_base + ne > O.e_cap) {         // edge pool full: the host grows it, runs the read again
                O.status[self] = OVF_POOL;
                const unsigned k = atomicAdd(next_count, 1u);
                next_list[k] = self;
            } else {
                O.status[self] = OVF_NONE;
                O.num_B[self] = uint16_t(nb);
                O.num_F[self] = uint16_t(nf);
                O.olp_B[self] = sb[0].olp;
                O.olp_F[self] = sb[1].olp;
                O.edge_src[self] = s_base;
            }
        }
        __syncthreads();
        const unsigned long long base = s_base;
        if (base + ne <= O.e_cap) {
            for (int e = tid; e < ne; e += T) {
                const uint32_t mt = e_meta[e];
                O.e_dest[base + e] = e_id[e];
                O.e_trans[base + e] = e_trans[e];
                O.e_len[base + e] = uint16_t(meta_len(mt));
                O.e_type[base + e] = uint8_t(meta_type(mt));
            }
        }
        __syncthreads();
    }
    add_probes(O, probes);
}

// reads with a side beyond `highest` candidates: to the next list
__global__ void k_block_beyond(const idx_t* list, unsigned count, const BlockSide* sides, unsigned highest, idx_t* next_list,
                               unsigned* next_count) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const BlockSide a = sides[2 * i], b = sides[2 * i + 1];
    if (max(a.olp ? a.m : 0u, b.olp ? b.m : 0u) > highest) next_list[atomicAdd(next_count, 1u)] = list[i];
}

constexpr int kBlockThreads = 256;

struct BlockSmem {      // a CTA's region of the global variant (offsets in bytes)
    size_t words, ids, metas, cnts, elist, e_ids, e_metas, e_trans, groups, prefs, read, bytes;
    size_t perm0, perm1, info;      // the sorted reduction's order and walk arrays
    int cap;            // candidates a side (and B-side edges kept while the F side is reduced)
    int nw;             // continuation words per candidate
};

// bytes a candidate takes (continuation words, read id, meta, counter, emitted list, B-side edge, two
// order arrays and the walk's array) and the fixed part (both sides' candidate
// groups, their prefix sums, the read)
size_t block_per_cand(int L, int t) {
    return size_t((L - t + 31) / 32) * 8 + sizeof(idx_t) + 4 + 4 + 4 + sizeof(idx_t) + 4 + 4 + 12;
}
size_t block_fixed(int L, int t) {
    const int M = L - t;
    return size_t(2) * size_t(2 * M) * sizeof(Cand) + size_t(2 * M + 1) * sizeof(unsigned) +
           size_t((L + 15) / 16) * sizeof(uint32_t) + 16 * 16;
}

BlockSmem block_smem_layout(int L, int t, size_t budget) {
    BlockSmem b{};
    const int M = L - t;
    b.nw = (M + 31) / 32;
    const size_t groups = size_t(2) * size_t(2 * M) * sizeof(Cand);
    const size_t prefs = size_t(2 * M + 1) * sizeof(unsigned);
    const size_t read = size_t((L + 15) / 16) * sizeof(uint32_t);
    const size_t per = block_per_cand(L, t);
    const size_t fixed = block_fixed(L, t);
    int cap = budget > fixed ? int(std::min<size_t>((budget - fixed) / per, 65535)) : 0;
    cap &= ~31;
    b.cap = cap;
    size_t o = 0;
    auto take = [&](size_t n) {
        const size_t r = o;
        o += (n + 15) & ~size_t(15);
        return r;
    };
    b.words = take(size_t(cap) * size_t(b.nw) * 8);
    b.ids = take(size_t(cap) * sizeof(idx_t));
    b.e_ids = take(size_t(cap) * sizeof(idx_t));
    b.metas = take(size_t(cap) * 4);
    b.cnts = take(size_t(cap) * 4);
    b.elist = take(size_t(cap) * 4);
    b.e_metas = take(size_t(cap) * 4);
    b.e_trans = take(size_t(cap) * 4);
    b.groups = take(groups);
    b.prefs = take(prefs);
    b.read = take(read);
    b.perm0 = take(size_t(cap) * 4);
    b.perm1 = take(size_t(cap) * 4);
    b.info = take(size_t(cap) * 4);
    b.bytes = o;
    return b;
}

constexpr int kBlockMaxWords = 8;       // continuation words a candidate (L - t <= 256)
// the digit counts' index with one pad word after every 16, so that a thread summing 16
// consecutive counts and its neighbours hit different banks
__device__ __forceinline__ int block_pad(int f) { return f + (f >> 4); }

// 4-bit digit q (0 = least significant) of candidate c's sort key: the continuation words (word 0
// most significant), then the continuation length (16 bits), then the read id.
__device__ __forceinline__ unsigned block_digit(const uint64_t* cw, int cap, int nw, const idx_t* cid,
                                                const uint32_t* cmeta, int L, int c, int q) {
    constexpr int kIdDigits = 2 * int(sizeof(idx_t));
    if (q < kIdDigits) return unsigned(uint64_t(cid[c]) >> (4 * q)) & 15u;
    q -= kIdDigits;
    if (q < 4) return (unsigned(L - meta_len(cmeta[c])) >> (4 * q)) & 15u;
    q -= 4;
    return unsigned(cw[size_t(nw - 1 - q / 16) * cap + c] >> (4 * (q % 16))) & 15u;
}

// One side's reduction by sorting, for the global-memory block tier (m up to 32768 candidates,
// where the m x m pair tests cost too much).  The candidates are ordered by (continuation, read id)
// with a stable LSD radix sort on 4-bit digits of (continuation words, length, read id): each
// thread counts and then places one contiguous run of the current order, and a digit that is the
// same for every candidate skips its placing.  Comparing the words (zero past each continuation's
// end) and then the length is the order in which a continuation precedes its extensions, so the
// candidates whose continuation starts with a given one follow it contiguously.  One walk then
// decides what the pair tests decide: a run of equal continuations with no earlier prefix among
// them is uncovered, the candidates after it that extend it are covered, trans = the run plus its
// extensions, and the run's second-kind candidates yield when a first-kind one is in it.  The
// emitted candidates come out in sorted order, which is the DFS order; they are written as the
// pair version writes them (B side: e_id/e_meta/e_trans by rank; F side: elist by rank, ccnt[c] =
// rank).  Returns the number emitted (in thread 0).
__device__ int block_sorted_side(int m, int L, int nw, int cap, const uint64_t* cw, const idx_t* cid,
                                 const uint32_t* cmeta, uint32_t* perm0, uint32_t* perm1, uint32_t* info,
                                 unsigned* scnt, unsigned* s_misc, int first_kind, idx_t self, int side,
                                 idx_t* e_id, uint32_t* e_meta, int32_t* e_trans, uint32_t* elist, uint32_t* ccnt) {
    constexpr int T = kBlockThreads;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int per = (m + T - 1) / T;
    const int b0 = min(m, tid * per), b1 = min(m, b0 + per);
    for (int i = tid; i < m; i += T) perm0[i] = uint32_t(i);
    uint32_t* src = perm0;
    uint32_t* dst = perm1;
    const int digits = 2 * int(sizeof(idx_t)) + 4 + 16 * nw;
    unsigned* s_wsum = s_misc;             // [T / 32]
    unsigned* s_dstart = s_misc + 8;       // [17]
    // which key bits differ between candidates: each key XOR candidate 0's, OR-reduced (id, length,
    // words); a digit whose bits never differ needs no pass at all
    unsigned long long* s_diff = reinterpret_cast<unsigned long long*>(s_misc + 26);   // [2 + nw]
    if (tid < 2 + nw) s_diff[tid] = 0;
    __syncthreads();
    {
        unsigned long long did = 0, dlen = 0, dw[kBlockMaxWords];
        #pragma unroll
        for (int w = 0; w < kBlockMaxWords; ++w) dw[w] = 0;
        const unsigned long long id0 = uint64_t(cid[0]), len0 = unsigned(L - meta_len(cmeta[0]));
        for (int c = tid; c < m; c += T) {
            did |= uint64_t(cid[c]) ^ id0;
            dlen |= unsigned(L - meta_len(cmeta[c])) ^ len0;
            #pragma unroll
            for (int w = 0; w < kBlockMaxWords; ++w)
                if (w < nw) dw[w] |= cw[size_t(w) * cap + c] ^ cw[size_t(w) * cap];
        }
        if (did) atomicOr(&s_diff[0], did);
        if (dlen) atomicOr(&s_diff[1], dlen);
        #pragma unroll
        for (int w = 0; w < kBlockMaxWords; ++w)
            if (w < nw && dw[w]) atomicOr(&s_diff[2 + w], dw[w]);
    }
    __syncthreads();
    for (int q = 0; q < digits; ++q) {
        {   // the digit's bits in the OR of differences: zero means every candidate has the same digit
            constexpr int kIdDigits = 2 * int(sizeof(idx_t));
            unsigned long long bits;
            if (q < kIdDigits) bits = s_diff[0] >> (4 * q);
            else if (q < kIdDigits + 4) bits = s_diff[1] >> (4 * (q - kIdDigits));
            else {
                const int r = q - kIdDigits - 4;
                bits = s_diff[2 + nw - 1 - r / 16] >> (4 * (r % 16));
            }
            if ((bits & 15ull) == 0) continue;
        }
        #pragma unroll
        for (int d = 0; d < 16; ++d) scnt[block_pad(d * T + tid)] = 0;
        for (int e = b0; e < b1; ++e)
            ++scnt[block_pad(block_digit(cw, cap, nw, cid, cmeta, L, int(src[e]), q) * T + tid)];
        __syncthreads();
        // exclusive scan of the 16 x T counts, digit-major: thread tid owns entries [16 tid, 16 tid + 16)
        unsigned mine = 0;
        #pragma unroll
        for (int j = 0; j < 16; ++j) mine += scnt[block_pad(16 * tid + j)];
        unsigned x = mine;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_wsum[wid] = x;
        __syncthreads();
        unsigned run = x - mine;
        for (int w = 0; w < wid; ++w) run += s_wsum[w];
        #pragma unroll
        for (int j = 0; j < 16; ++j) {
            const unsigned v = scnt[block_pad(16 * tid + j)];
            scnt[block_pad(16 * tid + j)] = run;
            run += v;
        }
        if ((16 * tid) % T == 0) s_dstart[(16 * tid) / T] = run - mine;   // the digit's first place
        if (tid == 0) s_dstart[16] = unsigned(m);
        __syncthreads();
        bool trivial = false;
        #pragma unroll
        for (int d = 0; d < 16; ++d) trivial |= s_dstart[d + 1] - s_dstart[d] == unsigned(m);
        if (!trivial) {
            for (int e = b0; e < b1; ++e) {
                const uint32_t c = src[e];
                dst[scnt[block_pad(block_digit(cw, cap, nw, cid, cmeta, L, int(c), q) * T + tid)]++] = c;
            }
            uint32_t* tmp = src;
            src = dst;
            dst = tmp;
        }
        __syncthreads();
    }
    // per position of the order: common prefix with the previous candidate (bases, capped at both
    // lengths) and the continuation length
    for (int k = tid; k < m; k += T) {
        const int c = int(src[k]);
        const int lc = L - meta_len(cmeta[c]);
        int lcp = 0;
        if (k > 0) {
            const int a = int(src[k - 1]);
            const int la = L - meta_len(cmeta[a]);
            lcp = 32 * nw;
            for (int w = 0; w < nw; ++w) {
                const uint64_t z = cw[size_t(w) * cap + a] ^ cw[size_t(w) * cap + c];
                if (z) {
                    lcp = 32 * w + (__clzll(z) >> 1);
                    break;
                }
            }
            lcp = min(lcp, min(la, lc));
        }
        info[k] = uint32_t(lcp) | (uint32_t(lc) << 16);
    }
    __syncthreads();
    int ne = 0;
    if (tid == 0) {
        for (int i = 0; i < m;) {
            const int lr = int(info[i] >> 16);
            int k = i + 1;
            while (k < m && int(info[k] & 0xffffu) >= lr && int(info[k] >> 16) == lr) ++k;
            const int eq_end = k;
            while (k < m && int(info[k] & 0xffffu) >= lr) ++k;
            const int32_t trans = int32_t(k - i);
            bool first_same = false;
            for (int j = i; j < eq_end; ++j) first_same |= meta_type(cmeta[src[j]]) == first_kind;
            for (int j = i; j < eq_end; ++j) {
                const int c = int(src[j]);
                if (cid[c] == self || (meta_type(cmeta[c]) != first_kind && first_same)) continue;
                if (side == 0) {
                    e_id[ne] = cid[c];
                    e_meta[ne] = cmeta[c];
                    e_trans[ne] = trans;
                } else {
                    elist[ne] = uint32_t(c) | (uint32_t(trans) << 16);
                    ccnt[c] = uint32_t(ne);
                }
                ++ne;
            }
            i = k;
        }
    }
    return ne;
}

// The block tier with its candidate arrays in a per-CTA region of `scratch` (global memory, cached in
// L1/L2), for sides of up to kBlockGlobalCap candidates; each side is reduced by block_sorted_side.
__global__ void __launch_bounds__(kBlockThreads) k_search_block_global(SearchArgs A, SearchOut O, const idx_t* list,
                                                                       const unsigned* list_count, BlockSmem lay,
                                                                       idx_t* next_list, unsigned* next_count,
                                                                       unsigned char* scratch) {
    extern __shared__ __align__(16) unsigned char smem_dyn[];
    unsigned char* smem = scratch + size_t(blockIdx.x) * lay.bytes;
    uint64_t* cw = reinterpret_cast<uint64_t*>(smem + lay.words);
    uint32_t* perm0 = reinterpret_cast<uint32_t*>(smem + lay.perm0);
    uint32_t* perm1 = reinterpret_cast<uint32_t*>(smem + lay.perm1);
    uint32_t* sinfo = reinterpret_cast<uint32_t*>(smem + lay.info);
    unsigned* scnt = reinterpret_cast<unsigned*>(smem_dyn);              // 16 x 256 counts, padded
    unsigned* smisc = scnt + 16 * kBlockThreads + 16 * kBlockThreads / 16;
    idx_t* cid = reinterpret_cast<idx_t*>(smem + lay.ids);
    uint32_t* cmeta = reinterpret_cast<uint32_t*>(smem + lay.metas);
    uint32_t* ccnt = reinterpret_cast<uint32_t*>(smem + lay.cnts);
    uint32_t* elist = reinterpret_cast<uint32_t*>(smem + lay.elist);
    idx_t* e_id = reinterpret_cast<idx_t*>(smem + lay.e_ids);
    uint32_t* e_meta = reinterpret_cast<uint32_t*>(smem + lay.e_metas);
    int32_t* e_trans = reinterpret_cast<int32_t*>(smem + lay.e_trans);
    Cand* grp = reinterpret_cast<Cand*>(smem + lay.groups);
    unsigned* pref = reinterpret_cast<unsigned*>(smem + lay.prefs);
    uint32_t* rdw = reinterpret_cast<uint32_t*>(smem + lay.read);
    __shared__ int s_n[2][2];
    __shared__ int32_t s_olp[2];
    __shared__ int s_ok, s_cnt[2];
    __shared__ unsigned long long s_base;
    const int tid = threadIdx.x;
    const int L = A.L, M = L - A.t, cap = lay.cap, nw = lay.nw;
    const unsigned count = *list_count;
    Tally probes;
    for (unsigned item = blockIdx.x; item < count; item += gridDim.x) {
        const idx_t self = list[item];
        if (tid == 0) {
            load_read(A, self, rdw, 1, probes);
            s_ok = 1;
        }
        __syncthreads();
        // the candidate groups of side B (thread 0) and side F (thread 32)
        if (tid == 0 || tid == 32) {
            const int side = tid ? 1 : 0;
            ReadView rd{rdw, 1};
            int n[2];
            int32_t olp = 0;
            chain_pair(A, A.fm, rd, side ? PQ_FB : PQ_BF, side ? PQ_FF : PQ_BB, n, olp, probes,
                       SlotsStack{grp + size_t(side) * 2 * M, M});
            s_n[side][0] = n[0];
            s_n[side][1] = n[1];
            s_olp[side] = olp;
        }
        __syncthreads();
        for (int side = 0; side < 2; ++side) {
            if (tid == 0) s_cnt[side] = 0;
            if (s_olp[side] == 0) {      // src/string_graph.c:824, 828
                __syncthreads();
                continue;
            }
            const int n0 = s_n[side][0], ng = n0 + s_n[side][1];
            const Cand* g = grp + size_t(side) * 2 * M;
            if (tid == 0) {       // group sizes are index-wide: summed in 64 bits, stopped past cap
                unsigned long long s = 0;
                for (int i = 0; i < ng && s <= (unsigned long long)cap; ++i) {
                    const Cand& c = g[i < n0 ? i : M + (i - n0)];
                    pref[i] = unsigned(s);
                    s += (unsigned long long)(c.uu - c.ll) + 1ull;
                }
                pref[ng] = unsigned(s);
                if (s > (unsigned long long)cap) s_ok = 0;
            }
            __syncthreads();
            if (!s_ok) break;
            const int m = int(pref[ng]);
            // every candidate's read id and continuation
            for (int i = tid; i < m; i += kBlockThreads) {
                int lo = 0, hi = ng - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (pref[mid] <= unsigned(i)) lo = mid;
                    else hi = mid - 1;
                }
                const Cand& c = g[lo < n0 ? lo : M + (lo - n0)];
                const idx_t row = c.ll + idx_t(unsigned(i) - pref[lo]);
                const FmView& fb = A.fm[cand_index(c.type)];
                const idx_t rp = read_of(__ldg(fb.sa + row), A.dl);
                const int d = int(c.len), len = L - d;
                const bool fwd = cand_index(c.type) == 1;
                const uint64_t* pk = A.fm[fwd ? 0 : 1].pk;
                const size_t pos = size_t(rp) * L + size_t(d);
                const uint64_t flip = fwd ? 0 : ~uint64_t(0);
                int used = 0;
                for (int w = 0; w < nw; ++w) {
                    const int left = len - 32 * w;
                    uint64_t x = 0;
                    if (left > 0) {
                        x = (text_window(pk, pos + 32 * w) ^ flip) & top_mask(left < 32 ? left : 32);
                        used = w + 1;
                    }
                    cw[size_t(w) * cap + i] = x;
                }
                probes.add(2, 1 + (used ? sectors_of(pk + (pos >> 5),
                                                     8 * ((((pos + 32 * (used - 1)) >> 5) - (pos >> 5)) + 2))
                                        : 0));
                cid[i] = rp;
                cmeta[i] = pack_meta(d, c.type);
            }
            __syncthreads();
            const int first_kind = side ? PQ_FB : PQ_BF;
            const int nsorted = block_sorted_side(m, L, nw, cap, cw, cid, cmeta, perm0, perm1, sinfo, scnt, smisc, first_kind,
                                                  self, side, e_id, e_meta, e_trans, elist, ccnt);
            if (tid == 0) s_cnt[side] = nsorted;
            __syncthreads();
        }
        if (!s_ok) {             // more candidates than fit: the next tier
            if (tid == 0) {
                const unsigned k = atomicAdd(next_count, 1u);
                next_list[k] = self;
            }
            __syncthreads();
            continue;
        }
        const int nb = s_cnt[0], nf = s_cnt[1], ne = nb + nf;
        if (tid == 0) {
            s_base = ne ? atomicAdd(O.e_count, (unsigned long long)ne) : 0ull;
            if (s_base + ne > O.e_cap) {         // edge pool full: the host grows it, runs the read again
                O.status[self] = OVF_POOL;
                const unsigned k = atomicAdd(next_count, 1u);
                next_list[k] = self;
            } else {
                O.status[self] = OVF_NONE;
                O.num_B[self] = uint16_t(nb);
                O.num_F[self] = uint16_t(nf);
                O.olp_B[self] = s_olp[0];
                O.olp_F[self] = s_olp[1];
                O.edge_src[self] = s_base;
            }
        }
        __syncthreads();
        const unsigned long long base = s_base;
        if (base + ne <= O.e_cap) {
            for (int e = tid; e < nb; e += kBlockThreads) {
                O.e_dest[base + e] = e_id[e];
                O.e_trans[base + e] = e_trans[e];
                O.e_len[base + e] = uint16_t(meta_len(e_meta[e]));
                O.e_type[base + e] = uint8_t(meta_type(e_meta[e]));
            }
            for (int i = tid; i < nf; i += kBlockThreads) {       // the F side's candidates are still in place
                const uint32_t v = elist[i];
                const int c = int(v & 0xffff);
                const unsigned long long q = base + nb + ccnt[c];
                O.e_dest[q] = cid[c];
                O.e_trans[q] = int32_t(v >> 16);
                O.e_len[q] = uint16_t(meta_len(cmeta[c]));
                O.e_type[q] = uint8_t(meta_type(cmeta[c]));
            }
        }
        __syncthreads();
    }
    add_probes(O, probes);
}

constexpr unsigned kWalkBatch = 8192;       // reads walked (and then reduced) at a time

template <int CAP, int T>
static int block_ctas(unsigned count) {
    int dev = 0, sms = 152, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t allowed = allow_smem<block_smem_bytes(CAP)>(k_search_block<CAP, T>);
    if (allowed != cudaSuccess) cudaGetLastError();         // the launch reports it
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_search_block<CAP, T>, T, block_smem_bytes(CAP));
    if (e != cudaSuccess) cudaGetLastError();
    return int(std::min<unsigned>(count, unsigned(sms * (e == cudaSuccess && per > 0 ? per : 1))));
}

// queue counters, walked sides, their groups, and the CTAs' regions: one area, since the three sizes
// run one after the other
static size_t block_layout(int L, int t, unsigned count, size_t (&o)[4]) {
    const unsigned nb = std::min(count, kWalkBatch);
    const int M = L - t, nw = (M + 31) / 32;
    const size_t region = std::max({size_t(block_ctas<kBlockSmall, 256>(nb)) * block_region_bytes(kBlockSmall, nw),
                                    size_t(block_ctas<kBlockMid, 512>(nb)) * block_region_bytes(kBlockMid, nw),
                                    size_t(block_ctas<kBlockLarge, 512>(nb)) * block_region_bytes(kBlockLarge, nw)});
    const size_t part[4] = {256, size_t(2 * nb) * sizeof(BlockSide), size_t(2 * nb) * size_t(2 * M) * sizeof(Cand), region};
    size_t used = 0;
    for (int i = 0; i < 4; ++i) {
        o[i] = used;
        used += (part[i] + 255) & ~size_t(255);
    }
    return used;
}

size_t block_scratch_bytes(int L, int t, unsigned count) {
    size_t o[4];
    return block_layout(L, t, count, o);
}

cudaError_t search_block(const SearchArgs& a, const SearchOut& o, const idx_t* list, unsigned count, void* scratch,
                         size_t scratch_bytes, idx_t* next_list, unsigned* next_count, cudaStream_t st) {
    size_t at[4];
    if (!count) return cudaSuccess;
    if (scratch_bytes < block_layout(a.L, a.t, count, at)) return cudaErrorInvalidValue;
    char* p = static_cast<char*>(scratch);
    unsigned* next = reinterpret_cast<unsigned*>(p + at[0]);
    BlockSide* sides = reinterpret_cast<BlockSide*>(p + at[1]);
    Cand* groups = reinterpret_cast<Cand*>(p + at[2]);
    const size_t rd = size_t((a.L + 15) / 16) * kWalkThreads * 4;
    if (rd > kMaxSmem) return cudaErrorInvalidValue;
    cudaError_t e = allow_smem<kMaxSmem>(k_block_walk);
    if (e != cudaSuccess) return e;
    for (unsigned b = 0; b < count; b += kWalkBatch) {
        const unsigned nb = std::min(count - b, kWalkBatch);
        e = cudaMemsetAsync(next, 0, 256, st);
        if (e != cudaSuccess) return e;
        k_block_walk<<<(2 * nb + kWalkThreads - 1) / kWalkThreads, kWalkThreads, rd, st>>>(a, o, list + b, nb, groups, sides);
        e = cudaGetLastError();                             // the next kernels index by what this leaves
        if (e != cudaSuccess) return e;
        note_launch();
        unsigned char* region = reinterpret_cast<unsigned char*>(p + at[3]);
        k_search_block<kBlockSmall, 256><<<block_ctas<kBlockSmall, 256>(nb), 256, block_smem_bytes(kBlockSmall), st>>>(
            a, o, list + b, nb, groups, sides, next, region, 0, kBlockSmall, next_list, next_count);
        k_search_block<kBlockMid, 512><<<block_ctas<kBlockMid, 512>(nb), 512, block_smem_bytes(kBlockMid), st>>>(
            a, o, list + b, nb, groups, sides, next + 1, region, kBlockSmall + 1, kBlockMid, next_list, next_count);
        k_search_block<kBlockLarge, 512><<<block_ctas<kBlockLarge, 512>(nb), 512, block_smem_bytes(kBlockLarge), st>>>(
            a, o, list + b, nb, groups, sides, next + 2, region, kBlockMid + 1, kBlockLarge, next_list, next_count);
        for (int i = 0; i < 3; ++i) note_launch();
        k_block_beyond<<<(nb + 255) / 256, 256, 0, st>>>(list + b, nb, sides, kBlockLarge, next_list, next_count);
        note_launch();
    }
    return cudaGetLastError();
}

// The same tier with the candidate arrays in global memory: kBlockGlobalCap candidates a side, one
// region of block_global_bytes / blocks bytes per CTA.
constexpr int kBlockGlobalCap = 32768;

int block_global_blocks(unsigned count) {
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const unsigned most = unsigned(sms) * 2;
    return int(count < most ? count : most);
}

BlockSmem block_global_layout(int L, int t) {
    return block_smem_layout(L, t, block_per_cand(L, t) * kBlockGlobalCap + block_fixed(L, t));
}
// the global variant's dynamic shared memory: the sort's 16 x kBlockThreads digit counts and a
// few words of scan state
constexpr size_t kBlockSortSmem = (16 * kBlockThreads + 16 * kBlockThreads / 16 + 64) * sizeof(unsigned);

size_t block_global_bytes(int L, int t, int blocks) { return size_t(blocks) * block_global_layout(L, t).bytes; }

cudaError_t search_block_global(const SearchArgs& a, const SearchOut& o, const idx_t* list, const unsigned* count,
                                unsigned count_host, int blocks, void* scratch, size_t scratch_bytes,
                                idx_t* next_list, unsigned* next_count, cudaStream_t st) {
    if (!count_host || blocks <= 0) return cudaSuccess;
    const BlockSmem lay = block_global_layout(a.L, a.t);
    if (scratch_bytes < size_t(blocks) * lay.bytes) return cudaErrorInvalidValue;
    k_search_block_global<<<blocks, kBlockThreads, kBlockSortSmem, st>>>(a, o, list, count, lay, next_list, next_count,
                                                                        static_cast<unsigned char*>(scratch));
    note_launch();
    return cudaGetLastError();
}

// Heavy tier: the fast kernel's DFS with 32 times the stack, 4 times the level width and 256
// levels, over a list of reads (the ones the fast tier could not hold: low-complexity sequence
// gives thousands of candidates a side).  Its own overflow goes to the wide tier.
constexpr int kHeavyCap = 16384, kHeavyFrames = 256, kHeavyPMax = 512;

size_t heavy_scratch_bytes(int L, int t, int blocks, int ebcap) {
    return scratch_layout(L - t, size_t(blocks) * kWarpsPerCta, ebcap, nullptr, nullptr, kHeavyCap, kHeavyFrames,
                          kHeavyPMax);
}

// A step of a warp takes as long as the intervals of all its reads, so few reads are spread over up to 512
// warps (8 MB of scratch each), 4 reads a warp or more: 3.8 thousand run reads of 320 bases at t = 30 took
// 600 ms with 32 a warp, now 288.
static int heavy_reads(unsigned count) { return int(std::min(32u, std::max(4u, (count + 511) / 512))); }
int heavy_blocks(unsigned count) {
    const unsigned per = unsigned(heavy_reads(count)), warps = (count + per - 1) / per;
    return int(std::min((warps + kWarpsPerCta - 1) / kWarpsPerCta, 152u * 2));
}

cudaError_t search_heavy(const SearchArgs& a, const SearchOut& o, const idx_t* list, const unsigned* count, unsigned count_host, int blocks,
                         void* scratch, size_t scratch_bytes, int ebcap, cudaStream_t st) {
    WarpScratch S;
    if (scratch_bytes < scratch_layout(a.L - a.t, size_t(blocks) * kWarpsPerCta, ebcap, scratch, &S, kHeavyCap,
                                       kHeavyFrames, kHeavyPMax))
        return cudaErrorInvalidValue;
    const int words = (a.L + 15) / 16;
    const size_t smem = size_t(words) * 32 * kWarpsPerCta * sizeof(uint32_t);
    SearchQueue Q{};
    Q.read_list = list;
    Q.list_count = count;
    Q.per = unsigned(heavy_reads(count_host));
    Q.dfs_max = kHeavyCap;
    // static shared memory (~46 KB) plus the reads: past the 48 KB a launch may take unasked
    constexpr size_t kReadSmem = 180 * 1024;            // reads of up to 5760 bases
    if (smem > kReadSmem) return cudaErrorInvalidValue;
    cudaError_t e = lam_words(a.L - a.t) == 2
        ? allow_smem<kReadSmem>(k_search_fast<2, kHeavyCap, kHeavyFrames, kHeavyPMax>)
        : allow_smem<kReadSmem>(k_search_fast<kLamWords, kHeavyCap, kHeavyFrames, kHeavyPMax>);
    if (e != cudaSuccess) return e;
    if (lam_words(a.L - a.t) == 2)
        k_search_fast<2, kHeavyCap, kHeavyFrames, kHeavyPMax><<<blocks, 32 * kWarpsPerCta, smem, st>>>(a, o, S, Q);
    else
        k_search_fast<kLamWords, kHeavyCap, kHeavyFrames, kHeavyPMax><<<blocks, 32 * kWarpsPerCta, smem, st>>>(a, o, S,
                                                                                                            Q);
    note_launch();
    return cudaGetLastError();
}

size_t queue_scratch_bytes(int M_max, size_t nwarps, int ebcap, bool lean) {
    return lean ? lean_layout(M_max, nwarps, ebcap, nullptr, nullptr) : scratch_layout(M_max, nwarps, ebcap, nullptr, nullptr);
}

cudaError_t search_fast_queue(const SearchQueue& queue, int L_max, int M_max, int blocks, void* scratch,
                              size_t scratch_bytes, int ebcap, cudaStream_t st) {
    const size_t nwarps = size_t(blocks) * kWarpsPerCta;
    WarpScratch S;
    if (scratch_bytes < scratch_layout(M_max, nwarps, ebcap, scratch, &S)) return cudaErrorInvalidValue;
    const int words = (L_max + 15) / 16;
    size_t smem = size_t(words) * 32 * kWarpsPerCta * sizeof(uint32_t);
    SearchQueue q = queue;
    q.per = 32;
    q.dfs_max = kTaskCap;
    SearchArgs a{};
    SearchOut o{};
    if (lam_words(M_max) == 2) k_search_fast<2, kTaskCap, kTaskFrames, kPMax><<<blocks, 32 * kWarpsPerCta, smem, st>>>(a, o, S, q);
    else k_search_fast<kLamWords, kTaskCap, kTaskFrames, kPMax><<<blocks, 32 * kWarpsPerCta, smem, st>>>(a, o, S, q);
    note_launch();
    return cudaGetLastError();
}

// Wide tier: the reference's own capacity bounds, scratch in global memory, one slot per thread, `lanes`
// of them a warp.  Threads of one warp go through their reads' DFS one after the other (they seldom stand at
// the same instruction), so a warp takes one read while there are warps: 13 run reads of 306 bases took
// 1.3 s in one warp, now 0.22.
__global__ void __launch_bounds__(64) k_search_wide(SearchArgs A, SearchOut O, const idx_t* list, unsigned count,
                                                    WideScratch W, int lanes) {
    extern __shared__ uint32_t s_reads[];
    __shared__ FmView s_fm[2];
    if (threadIdx.x < 2) s_fm[threadIdx.x] = A.fm[threadIdx.x];
    __syncthreads();
    const unsigned slot = (blockIdx.x * blockDim.x + threadIdx.x) / 32 * unsigned(lanes) + (threadIdx.x & 31u);
    Tally probes;
    if (int(threadIdx.x & 31u) < lanes && slot < unsigned(W.slots)) {
        Cand* stk = reinterpret_cast<Cand*>(W.stack) + size_t(slot) * W.stack_cap;
        Frame* fr = reinterpret_cast<Frame*>(W.frames) + size_t(slot) * W.frame_cap;
        EdgeRec* eb = reinterpret_cast<EdgeRec*>(W.edges) + size_t(slot) * W.edge_cap;
        for (unsigned i = slot; i < count; i += unsigned(W.slots)) {
            idx_t r = list[i];
            load_read(A, r, s_reads + threadIdx.x, blockDim.x, probes);
            ReadView rd{s_reads + threadIdx.x, int(blockDim.x)};
            ReadResult R = search_read(A, s_fm, r, rd, stk, int(W.stack_cap), fr, int(W.frame_cap), eb,
                                       int(W.edge_cap), probes);
            if (R.status == OVF_STACK || R.status == OVF_LEVELS) R.status = ERR_CAP;
            if (R.status == ERR_CAP || R.status == ERR_TOO_MANY || R.status == OVF_EDGES) {
                O.status[r] = uint8_t(R.status == OVF_EDGES ? ERR_CAP : R.status);
                continue;
            }
            // pool overflow is reported through status and the host grows the pool and retries
            unsigned long long base = 0;
            if (R.ne) {
                base = atomicAdd(O.e_count, (unsigned long long)R.ne);
                if (base + R.ne > O.e_cap) { O.status[r] = OVF_POOL; continue; }
                for (int e = 0; e < R.ne; ++e) {
                    O.e_dest[base + e] = eb[e].dest;
                    O.e_trans[base + e] = eb[e].trans;
                    O.e_len[base + e] = eb[e].len;
                    O.e_type[base + e] = eb[e].type;
                }
            }
            O.status[r] = OVF_NONE;
            O.num_B[r] = uint16_t(R.nB);
            O.num_F[r] = uint16_t(R.nF);
            O.olp_B[r] = R.olpB;
            O.olp_F[r] = R.olpF;
            O.edge_src[r] = base;
        }
    }
    if (probes.probes) atomicAdd(O.probes, (unsigned long long)probes.probes);
    if (probes.sectors) atomicAdd(O.sectors, (unsigned long long)probes.sectors);
}

size_t wide_slot_bytes(int L) {
    size_t cap = size_t(2 * L) * size_t(2 * L);
    return cap * sizeof(Cand) + size_t(L + 2) * sizeof(Frame) + size_t(2 * 65535 + 2) * sizeof(EdgeRec);
}

cudaError_t search_wide(const SearchArgs& a, const SearchOut& o, const idx_t* list, unsigned count,
                        const WideScratch& ws, cudaStream_t st) {
    if (!count) return cudaSuccess;
    const int tpb = 64;
    const int words = (a.L + 15) / 16;
    size_t smem = size_t(words) * tpb * sizeof(uint32_t);
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int lanes = std::min(32, (ws.slots + 16 * sms - 1) / (16 * sms));
    const int warps = (ws.slots + lanes - 1) / lanes;
    { k_search_wide<<<(warps + 1) / 2, tpb, smem, st>>>(a, o, list, count, ws, lanes); note_launch(); }
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------ CSR assembly

// exclusive scan of 64-bit counts: tiles of 1024 per CTA (3 passes)
// of `in`, or of the reads' edge counts (the last entry is none)
struct EdgeCounts {
    const uint16_t *nB, *nF;
    size_t reads;
    __device__ unsigned long long operator[](size_t i) const { return i < reads ? (unsigned long long)nB[i] + nF[i] : 0ull; }
};
template <class In>
__global__ void k_scan_tiles(In in, size_t n, unsigned long long* out, unsigned long long* tile_sums) {
    __shared__ unsigned long long warp_sum[32];
    const size_t tile = blockIdx.x;
    const size_t i = tile * 1024 + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long v = i < n ? in[i] : 0, x = v;
    #pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        unsigned long long w = warp_sum[lane], z = w;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long y = __shfl_up_sync(0xffffffffu, z, o);
            if (lane >= o) z += y;
        }
        warp_sum[lane] = z - w;
        if (lane == 31 && tile_sums) tile_sums[tile] = z;
    }
    __syncthreads();
    if (i < n) out[i] = warp_sum[wid] + x - v;
}

__global__ void k_scan_add(unsigned long long* out, size_t n, const unsigned long long* tile_off) {
    const size_t i = size_t(blockIdx.x) * 1024 + threadIdx.x;
    if (i < n) out[i] += tile_off[blockIdx.x];
}

template <class In>
static void scan_u64(In in, size_t n, unsigned long long* out, unsigned long long* tmp,
                     cudaStream_t st) {
    if (n == 0) return;
    size_t tiles = (n + 1023) / 1024;
    if (tiles == 1) {
        { k_scan_tiles<<<1, 1024, 0, st>>>(in, n, out, nullptr); note_launch(); }
        return;
    }
    unsigned long long* sums = tmp;
    unsigned long long* sums_scan = tmp + tiles;
    { k_scan_tiles<<<unsigned(tiles), 1024, 0, st>>>(in, n, out, sums); note_launch(); }
    scan_u64<const unsigned long long*>(sums, tiles, sums_scan, tmp + 2 * tiles, st);
    { k_scan_add<<<unsigned(tiles), 1024, 0, st>>>(out, n, sums_scan); note_launch(); }
}

size_t assemble_tmp_bytes(idx_t num_reads) {
    size_t n = size_t(num_reads) + 1, total = 0;
    size_t t = (n + 1023) / 1024;
    while (t > 1) { total += 2 * t; t = (t + 1023) / 1024; }
    return (total + 64) * sizeof(unsigned long long);
}

// A warp copies the edges of 32 reads, an edge a lane whatever read it belongs to: a read of a thousand
// edges does not hold one thread, and the CSR arrays are written in whole sectors.  Bound by memory;
// with a thread a read, the 3,645 run reads of the 200 Mbp workload at 1/100 genome took 0.95 ms, now 0.37.
__global__ void k_gather_edges(const SearchOut O, idx_t n, const unsigned long long* off, idx_t* dest,
                               uint16_t* len, uint8_t* type, int32_t* trans) {
    const int lane = int(threadIdx.x & 31u);
    const size_t warps = size_t(gridDim.x) * blockDim.x / 32, nn = size_t(n);
    for (size_t r0 = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * 32; r0 < nn; r0 += warps * 32) {
        const size_t r = r0 + size_t(lane);
        const unsigned long long lo = off[r < nn ? r : nn], src = r < nn ? O.edge_src[r] : 0;
        const unsigned long long first = __shfl_sync(0xffffffffu, lo, 0), last = off[r0 + 32 < nn ? r0 + 32 : nn];
        for (unsigned long long e0 = first; e0 < last; e0 += 32) {
            const unsigned long long e = e0 + unsigned(lane);
            int q = 0;                                          // the last of the 32 reads to start at or before e
            #pragma unroll
            for (int w = 16; w; w >>= 1)
                if (__shfl_sync(0xffffffffu, lo, q + w) <= e) q += w;
            const unsigned long long s = __shfl_sync(0xffffffffu, src, q) + (e - __shfl_sync(0xffffffffu, lo, q));
            if (e < last) {
                dest[e] = O.e_dest[s];
                len[e] = O.e_len[s];
                type[e] = O.e_type[s];
                trans[e] = O.e_trans[s];
            }
        }
    }
}

cudaError_t assemble_counts_total(const SearchOut& o, idx_t num_reads, unsigned long long* out_off, void* scan_tmp,
                                  size_t scan_tmp_bytes, cudaStream_t st) {
    const size_t n = size_t(num_reads);
    if (scan_tmp_bytes < assemble_tmp_bytes(num_reads)) return cudaErrorInvalidValue;
    scan_u64(EdgeCounts{o.num_B, o.num_F, n}, n + 1, out_off, reinterpret_cast<unsigned long long*>(scan_tmp), st);
    return cudaGetLastError();
}

cudaError_t assemble_gather(const SearchOut& o, idx_t num_reads, const unsigned long long* off, idx_t* dest,
                            uint16_t* len, uint8_t* type, int32_t* trans, cudaStream_t st) {
    const size_t n = size_t(num_reads);
    unsigned g = unsigned(std::min<size_t>((n + 255) / 256 + 1, 152 * 32));
    if (n) { k_gather_edges<<<g, 256, 0, st>>>(o, idx_t(n), off, dest, len, type, trans); note_launch(); }
    return cudaGetLastError();
}

const size_t kCandBytes = sizeof(Cand);
const size_t kFrameBytes = sizeof(Frame);

}  // namespace pq
