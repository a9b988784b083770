// pq_sort.cuh — GPU suffix sort of read-bounded suffixes (internal).
#pragma once
#include "pq_common.cuh"

namespace pq {

// Suffix array of direction dir in the canonical order (suffix string with end-of-read lowest,
// then text position).  Returns 0 or a cudaError_t value.  cap (0: none) is the largest number of
// suffixes the caller wants sorted at a time: the sort then takes no more working memory than chunks
// of that size would (in chunks when one pass needs more), and returns cudaErrorNotSupported when a
// 6-base bucket exceeds it or the reads are longer than kChunkMaxLen (so do more than 2^31 - 1 suffixes of
// reads too long for the networks, with or without it).  When bwt_out is given it receives the BWT symbol (0 = `$`, 1..4) of
// every row, inside tmp (valid until tmp is reused), or nullptr when the sort went by prefix
// doubling.  pk_out (n/32 + 4 words), when given, receives the packed text of the direction (see
// pack_text) instead of tmp.  kt, when given, receives the table of kmer_k-mers (FmView::kt) and kx
// (n entries), when given beside it, every row's next bases (FmView::kx); *kmer_done tells whether
// the table is complete (else the caller builds it) and *kx_bases how many bases kx holds (0: none).
constexpr int kSortKeyBases = 14;           // longest k-mers of the table
constexpr int kChunkMaxLen = 268;           // longest reads sorted in chunks
size_t suffix_sort_tmp_bytes(size_t n, size_t num_reads, int L, size_t cap = 0);
int suffix_sort(const uint8_t* reads, idx_t num_reads, int L, int dir, idx_t* sa, size_t cap, void* tmp,
                size_t tmp_bytes, cudaStream_t st, const uint8_t** bwt_out = nullptr, uint64_t* pk_out = nullptr,
                idx_t* kt = nullptr, int kmer_k = 0, bool* kmer_done = nullptr, uint16_t* kx = nullptr, int* kx_bases = nullptr);

// Per-read seeds from a k-mer table (pq_index.cu).
cudaError_t read_seeds(const uint8_t* reads, idx_t num_reads, int L, int dir, int k, const idx_t* kt,
                       idx_t* start, idx_t* size, cudaStream_t st);

// Stable LSD radix sort of (key, value) pairs on the bits [lo_bit, hi_bit) of the key (K is
// uint32_t or uint64_t).  Buffers are ping-ponged; the sorted result ends in (*k0, *v0) (pointers
// may be swapped).  skip_trivial: first histogram every digit (one pass and a host round trip)
// and skip the digits that are constant over all keys; else run every digit pass.
template <class K, class V>
int radix_sort_pairs(K** k0, V** v0, K** k1, V** v1, size_t n, int lo_bit, int hi_bit,
                     void* tmp, size_t tmp_bytes, cudaStream_t st, bool skip_trivial = true);
size_t radix_tmp_bytes(size_t n);

// The text of direction dir packed 32 bases per 64-bit word, first base in the top bits
// (n/32 + 4 words; the last words are zero padding).
cudaError_t pack_text(const uint8_t* reads, size_t n, idx_t L, int dir, uint64_t* pk, cudaStream_t st);

}  // namespace pq
