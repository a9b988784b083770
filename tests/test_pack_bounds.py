"""The reversed text packed eight bases a step (pasqual_gb300/csrc/pq_pack.h): the right bases, and no word
that reaches outside the caller's read bytes, at every alignment and at both ends.  Host code, compiled
with the host compiler."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "pq_pack.h"
int main() {
    long bad = 0, outside = 0, unguarded = 0, words = 0, fast = 0;
    for (size_t L = 8; L <= 120; L += L < 40 ? 1 : 19)
        for (size_t nr = 1; nr <= 9; ++nr)
            for (size_t mis = 0; mis < 8; ++mis) {
                const size_t n = nr * L;
                std::vector<uint64_t> mem(n / 8 + 4);
                unsigned char* base = reinterpret_cast<unsigned char*>(mem.data()) + 8 + mis;
                for (size_t i = 0; i < n; ++i) base[i] = 1 + (i * 7 + i / 5 + L) % 4;
                const uintptr_t lo = reinterpret_cast<uintptr_t>(base), hi = lo + n;
                for (size_t p0 = 0; p0 + 32 <= n; p0 += 32) {
                    long out = 0;
                    auto word = [&](uintptr_t a) {
                        uint64_t v;
                        out += a < lo || a + 8 > hi;
                        std::memcpy(&v, reinterpret_cast<const void*>(a), 8);
                        return v;
                    };
                    const size_t r = p0 / L;
                    const uint64_t got = pq::pack_backward(lo, r, p0 - r * L, L, word);
                    uint64_t want = 0;
                    for (size_t p = p0; p < p0 + 32; ++p) want = want << 2 | (base[p / L * L + (L - 1 - p % L)] - 1u);
                    bad += got != want;
                    ++words;
                    unguarded += out;
                    if (pq::pack_inside(lo, n, p0, L)) { outside += out; ++fast; }
                }
            }
    printf("%ld words, %ld eight at a time, %ld wrong, %ld loads outside (%ld without the test)\n", words, fast, bad, outside, unguarded);
    return bad || outside || !unguarded || fast * 4 < words;
}
"""


def test_no_word_outside_the_reads(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host C++ compiler")
    (tmp_path / "h.cpp").write_text(HARNESS)
    exe = str(tmp_path / "h")
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wno-unknown-pragmas", "-I", os.path.join(ROOT, "pasqual_gb300", "csrc"),
                    str(tmp_path / "h.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
