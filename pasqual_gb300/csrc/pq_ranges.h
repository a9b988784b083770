// pq_ranges.h — ranges of elements described by the host for kernels that take them a tile at a time,
// and the host memory of the asynchronous copies that bring them to the device.  Host code only.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <deque>
#include <utility>
#include <vector>

namespace pq {

// Blocks of host memory that copies read until the stream has been waited for: a copy from pageable
// memory may still read its source after the call that enqueued it has returned.  `Wait` waits for the
// stream; it is called by wait() and, with blocks still held, at the end.
template <class Wait>
class HeldBlocks {
    Wait wait_;
    std::deque<std::vector<unsigned char>> blocks_;

public:
    explicit HeldBlocks(Wait w) : wait_(std::move(w)) {}
    HeldBlocks(const HeldBlocks&) = delete;
    HeldBlocks& operator=(const HeldBlocks&) = delete;
    ~HeldBlocks() {
        if (!blocks_.empty()) wait_();
    }
    unsigned char* take(size_t bytes) {
        blocks_.emplace_back(bytes);
        return blocks_.back().data();
    }
    auto wait() {
        const auto r = wait_();
        blocks_.clear();
        return r;
    }
    size_t held() const { return blocks_.size(); }
};

// One block for `count` ranges: starts and ends (64-bit), the exclusive scan of their tiles (count + 1),
// their offsets and shifts (32-bit).  Byte positions of the parts.
struct RangeBlock {
    size_t count;
    size_t ends() const { return 8 * count; }
    size_t tiles() const { return 16 * count; }
    size_t offs() const { return 20 * count + 4; }
    size_t shifts() const { return 24 * count + 4; }
    size_t bytes() const { return 28 * count + 4; }
};

// Fills such a block from ranges (start, end, off) and, with `shift`, their shifts; returns the tiles.
template <class Range>
unsigned fill_ranges(unsigned char* at, const Range* r, size_t count, const int* shift, size_t tile) {
    const RangeBlock b{count};
    unsigned tiles = 0;
    auto put = [&](size_t pos, auto v) { std::memcpy(at + pos, &v, sizeof v); };
    for (size_t i = 0; i < count; ++i) {
        put(8 * i, uint64_t(r[i].start));
        put(b.ends() + 8 * i, uint64_t(r[i].end));
        put(b.tiles() + 4 * i, tiles);
        put(b.offs() + 4 * i, int32_t(r[i].off));
        put(b.shifts() + 4 * i, int32_t(shift ? shift[i] : 0));
        tiles += unsigned((r[i].end - r[i].start + tile - 1) / tile);
    }
    put(b.tiles() + 4 * count, tiles);
    return tiles;
}

}  // namespace pq
