"""The index arithmetic by which the batched kernels find a tile's segment heads
(csrc/segment_search.h), compiled for the host and run over batches of up to
2^32 - 2 segments, the most the library takes: offsets are a formula, not memory.
Every search has to end within a few rounds, read entries of the batch only, and
leave an interval that holds the first offset at or past the tile's start.
"""
import subprocess

from gpuprefixsums_gb300 import build as B

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "segment_search.h"
using namespace gps;

// `segments` offsets, of which the first `low` are 0 and the others spread over (0, n].
struct Batch {
    uint64_t segments, low, n;
    uint64_t at(uint64_t i) const {
        if (i > segments) { printf("entry %llu of %llu\n", (unsigned long long)i, (unsigned long long)segments); exit(1); }
        return i < low ? 0 : 1 + (i - low) * (n - 1) / (segments - low + 1);
    }
    uint64_t first(uint64_t start) const {  // index of the first offset at or past it
        uint64_t lo = 0, hi = segments;
        while (lo < hi) {
            const uint64_t m = lo + (hi - lo) / 2;
            if (at(m) < start) lo = m + 1; else hi = m;
        }
        return lo;
    }
};

static void check(const Batch& b, OffsetInterval iv, uint64_t start, uint32_t probes, uint64_t most, const char* what) {
    int rounds = 0;
    while (iv.size() > most) {
        uint32_t below = 0;
        for (uint32_t p = 0; p < probes; ++p) {
            const uint32_t d = iv.probe(p, probes);
            if (d < iv.size() && b.at(uint64_t(iv.lo) + d) < start) ++below;
        }
        iv.narrow(below, probes);
        if (++rounds > 8) { printf("%s: no end\n", what); exit(1); }
    }
    const uint64_t want = b.first(start);
    // (Of equal offsets at the start, the first found will do.)
    const bool in = iv.lo <= want && want <= iv.hi;
    if (!(iv.lo <= iv.hi && iv.hi <= b.segments && (in || b.at(iv.lo) == start))) {
        printf("%s: %llu segments, %llu low, start %llu: [%llu, %llu] without %llu\n", what, (unsigned long long)b.segments,
               (unsigned long long)b.low, (unsigned long long)start, (unsigned long long)iv.lo, (unsigned long long)iv.hi,
               (unsigned long long)want);
        exit(1);
    }
}

int main() {
    const uint64_t counts[] = {1, 2, 255, 256, 257, 1023, 1024, 1025, 70000, 16777215, 16777217, 4000000000ull,
                               4294966270ull, 4294966271ull, 4294966272ull, 4294967038ull, 4294967039ull,
                               4294967040ull, 4294967293ull, 4294967294ull};
    const uint64_t n = 5000011;
    for (uint64_t c : counts)
        for (uint64_t low : {uint64_t(1), c / 2 + 1, c - c / 1000, c}) {
            const Batch b{c, low, n};
            for (uint64_t start : {uint64_t(1), uint64_t(4096), uint64_t(16384), uint64_t(2498560), n / 4096 * 4096}) {
                check(b, OffsetInterval{0, static_cast<uint32_t>(c)}, start, 256, 1024, "one tile per CTA");
                const OffsetSamples s(static_cast<uint32_t>(c));
                if (s.stride == 0 || s.count == 0 || s.count > 1024 || uint64_t(s.count) * s.stride <= c ||
                    uint64_t(s.count - 1) * s.stride > c) {
                    printf("samples of %llu segments: %u of stride %u\n", (unsigned long long)c, s.count, s.stride);
                    return 1;
                }
                uint32_t k = 0;  // the first sample past the start
                while (k < s.count && b.at(uint64_t(k) * s.stride) <= start) ++k;
                check(b, s.interval(k, static_cast<uint32_t>(c)), start, 32, 256, "units");
            }
        }
    return 0;
}
"""


def test_searches_of_up_to_the_most_segments(tmp_path):
    src, exe = tmp_path / "search.cpp", tmp_path / "search"
    src.write_text(PROGRAM)
    res = subprocess.run(["g++", "-std=c++17", "-O1", "-I", B.CSRC_DIR, "-o", str(exe), str(src)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-2000:]
