// pq_pack.h — eight bases at a time from the read bytes (codes 1..4) to the packed text's 2 bits each,
// first base in the top bits.  For device code and, with another way to load a word, for the host.
#pragma once

#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define PQ_HD __host__ __device__ __forceinline__
#else
#define PQ_HD inline
#endif

namespace pq {

// eight bytes of codes 1..4, the first base highest, as 16 bits
PQ_HD uint32_t pack8(uint64_t x) {
    x -= 0x0101010101010101ull;
    x = (x | (x >> 6)) & 0x000f000f000f000full;
    x = (x | (x >> 12)) & 0x000000ff000000ffull;
    return uint32_t((x | (x >> 24)) & 0xffffu);
}

// the eight bytes at address a, first byte lowest, from the aligned 8-byte words that hold them
template <class Word>
PQ_HD uint64_t load8(uintptr_t a, Word word) {
    const uintptr_t w = a & ~uintptr_t(7);
    const int s = 8 * int(a & 7);
    const uint64_t lo = word(w);
    return s ? (lo >> s) | (word(w + 8) << (64 - s)) : lo;
}

// The reversed reads' text from offset `off` of read r on, 32 bases of at least 8 a read: the eight of a
// step lie in one read, last first, or in the start of one and the end of the next.
template <class Word>
PQ_HD uint64_t pack_backward(uintptr_t reads, size_t r, size_t off, size_t L, Word word) {
    uint64_t v = 0;
    #pragma unroll
    for (int j = 0; j < 4; ++j) {
        const size_t k = L - off;                   // bases left in read r
        uint64_t x = load8(reads + r * L + (k < 8 ? 0 : k - 8), word);
        if (k < 8) x = (x << (64 - 8 * k)) | (load8(reads + (r + 2) * L - 8, word) >> (8 * k));
        v = (v << 16) | pack8(x);
        off += 8;
        if (off >= L) {
            off -= L;
            ++r;
        }
    }
    return v;
}

// Whether every word that pack_backward loads for the bases [p0, p0 + 32) of n lies within the n read
// bytes: always where they start and end on a word, else away from the ends (the bytes of a read and
// the one after it, rounded to words).
PQ_HD bool pack_inside(uintptr_t reads, size_t n, size_t p0, size_t L) {
    return p0 + 32 <= n && (reads % 8 == 0 || p0 >= L + 7) && ((reads + n) % 8 == 0 || p0 + 31 + L + 7 <= n);
}

}  // namespace pq
