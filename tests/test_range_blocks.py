"""The host blocks of the sort's copies to the device (pasqual_gb300/csrc/pq_ranges.h): a copy that reads
its source only when the stream is waited for still finds what it was given, however many ranges were
described in between, and the blocks end with a wait.  Host code, compiled with the host compiler."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <functional>
#include "pq_ranges.h"
struct Range { unsigned long long start, end; int off; };
int main() {
    std::vector<std::function<void()>> queue;           // a stream whose copies run when it is waited for
    int waits = 0, bad = 0;
    auto wait = [&] { ++waits; for (auto& f : queue) f(); queue.clear(); return 0; };
    const size_t tile = 100;
    std::vector<std::vector<unsigned char>> dev;
    std::vector<std::vector<Range>> given;
    std::vector<std::vector<int>> shifts;
    {
        pq::HeldBlocks<decltype(wait)> held(wait);
        auto describe = [&](size_t count, unsigned seed, bool with_shift) {
            std::vector<Range> r(count);
            std::vector<int> sh(count);
            for (size_t i = 0; i < count; ++i) {
                r[i].start = (unsigned long long)seed << 33 | i * 1000;
                r[i].end = r[i].start + 1 + (i * 37 + seed) % 950;
                r[i].off = int(i % 300);
                sh[i] = int((i + seed) % 60);
            }
            const pq::RangeBlock b{count};
            unsigned char* h = held.take(b.bytes());
            const unsigned tiles = pq::fill_ranges(h, r.data(), count, with_shift ? sh.data() : nullptr, tile);
            unsigned want = 0;
            for (auto& x : r) want += unsigned((x.end - x.start + tile - 1) / tile);
            bad += tiles != want;
            const size_t at = dev.size(), n = b.bytes();
            dev.emplace_back(n);
            queue.push_back([&dev, at, h, n] { std::memcpy(dev[at].data(), h, n); });
            given.push_back(r);
            shifts.push_back(with_shift ? sh : std::vector<int>(count, 0));
        };
        for (int round = 0; round < 3; ++round) {
            for (unsigned k = 0; k < 40; ++k) describe(1 + (k * 131 + round) % 4096, k + 1, k & 1);
            bad += held.held() != 40;
            if (round < 2) { held.wait(); bad += held.held() != 0; }
        }
    }                                                   // copies in flight: waited for at the end
    bad += waits != 3;
    for (size_t d = 0; d < dev.size(); ++d) {
        const size_t c = given[d].size();
        const pq::RangeBlock b{c};
        const unsigned char* p = dev[d].data();
        auto u64 = [&](size_t at) { unsigned long long v; std::memcpy(&v, p + at, 8); return v; };
        auto u32 = [&](size_t at) { unsigned v; std::memcpy(&v, p + at, 4); return v; };
        bad += b.tiles() % 4 || b.offs() % 4 || b.shifts() % 4 || b.shifts() + 4 * c != b.bytes();
        unsigned tiles = 0;
        for (size_t i = 0; i < c; ++i) {
            const Range& r = given[d][i];
            bad += u64(8 * i) != r.start || u64(b.ends() + 8 * i) != r.end || u32(b.tiles() + 4 * i) != tiles ||
                   int(u32(b.offs() + 4 * i)) != r.off || int(u32(b.shifts() + 4 * i)) != shifts[d][i];
            tiles += unsigned((r.end - r.start + tile - 1) / tile);
        }
        bad += u32(b.tiles() + 4 * c) != tiles;
    }
    printf("%zu blocks, %d bad\n", dev.size(), bad);
    return bad != 0;
}
"""


def test_sources_outlive_their_copies(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    (tmp_path / "h.cpp").write_text(HARNESS)
    exe = str(tmp_path / "h")
    subprocess.run([gxx, "-O1", "-g", "-fsanitize=address", "-std=c++17", "-I", os.path.join(ROOT, "pasqual_gb300", "csrc"),
                    str(tmp_path / "h.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


def test_the_sort_copies_from_no_other_memory():
    """more_splits enqueues every copy to the device from a held block."""
    src = open(os.path.join(ROOT, "pasqual_gb300", "csrc", "pq_sort.cu")).read()
    body = src[src.index("int more_splits("):src.index("struct SortOut")]
    assert body.count("cudaMemcpyHostToDevice") == body.count("held.take(") == 2
    assert body.count("cudaStreamSynchronize") == 1         # the one behind held.wait()
