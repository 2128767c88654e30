// Where a tile's segment heads begin in the offsets of a batch: index
// arithmetic shared by the batched kernels. A batch may have up to 2^32 - 2
// segments (most of them empty), so indices are compared as distances from the
// interval's start: neither a sum past its end nor a rounded-up division may wrap.
// (In 64 bits the search is as right and costs more: 2^26 compensated FP32 in 500
// segments 106.4 -> 107.6 us, like this 106.2-106.9; 2^26 u32 in 6 M segments 210, like this 208.)
// Compiles with a host compiler too.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GPS_HD __host__ __device__ __forceinline__
#else
#define GPS_HD inline
#endif

namespace gps {

// The first offset at or past a tile's start has an index in [lo, hi]: entries
// before lo lie below the start, entry hi, if there is one, does not. Probes of a
// non-empty interval:
struct OffsetInterval {
    uint32_t lo, hi;
    GPS_HD uint32_t size() const { return hi - lo; }
    // Distance from lo of the entry for probe i of `probes`; at size() or more, none.
    GPS_HD uint32_t probe(uint32_t i, uint32_t probes) const { return i * step(probes); }
    // The first `below` of the probes lie below the start.
    GPS_HD void narrow(uint32_t below, uint32_t probes) {
        const uint32_t s = step(probes), first = lo;
        const uint64_t end = static_cast<uint64_t>(below) * s;
        if (below != 0) lo = first + static_cast<uint32_t>(end) - s + 1;
        if (end < hi - first) hi = first + static_cast<uint32_t>(end);
    }

private:
    GPS_HD uint32_t step(uint32_t probes) const { return (size() - 1) / probes + 1; }
};

// Samples of the offsets: entries 0, stride, 2 * stride .. up to entry `segments`, at
// most 1024.
struct OffsetSamples {
    uint32_t stride, count;
    GPS_HD explicit OffsetSamples(uint32_t segments) : stride(segments / 1024 + 1), count(segments / stride + 1) {}
    // The interval that the first sample past the start, number `s`, leaves.
    GPS_HD OffsetInterval interval(uint32_t s, uint32_t segments) const {
        return OffsetInterval{s == 0 ? 0 : (s - 1) * stride, s < count ? s * stride : segments};
    }
};

}  // namespace gps
