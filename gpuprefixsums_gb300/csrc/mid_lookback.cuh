// Lookback of the one-tile-per-CTA kernels over integer sums: the scans of mid.cu and
// the counts of select.cu.
#pragma once
#include "tile_rows.cuh"

namespace gps {

// ------------------------------------------------------------ descriptors
// One 16-byte word per tile: {lo: the value (u32 or u64), hi: status:2 |
// launch number:62}. Zeroed memory reads "not ready". Tile t's
// word is word t * a.desc_stride of the region: launches of more than one
// group of tiles give each tile a 128-byte line of its own, since tiles that
// publish while others read the same line waited up to 3 us for a read.
constexpr uint64_t kTagMask = (1ull << 62) - 1;

struct MidDesc {
    __device__ static ptx::u64x2 pack(uint32_t status, uint64_t tag, uint64_t v) {
        ptx::u64x2 w;
        w.lo = v;
        w.hi = (static_cast<uint64_t>(status) << 62) | (tag & kTagMask);
        return w;
    }
    __device__ static uint32_t status(const ptx::u64x2& w, uint64_t tag) {
        return (w.hi & kTagMask) == (tag & kTagMask) ? static_cast<uint32_t>(w.hi >> 62) : kNotReady;
    }
};

// ---------------------------------------------------------------- lookback
// Tiles form groups of 32. A tile publishes its sum twice, at once: in its
// descriptor, and by an atomic addition to its group's sum, a 64-bit word with
// the number of tiles added so far above bit 40 (two such words for u64, one
// for each half of the values). The prefix of a tile is then the sums of the
// groups before, complete at a count of 32, and the descriptors of the tiles
// before in its own group: warp 0 polls these and the first 32 groups together, the
// next three warps 32 groups each, so every tile waits for one L2 round trip
// after the last tile before it has published.
//
// The group sums have two sets, which the launches that use them take in turn,
// counted in the plan's header; tile 0's CTA clears the other set for the next.
// Warp 0 reads the launch number and that count in one load and hands the count
// to the CTA through shared memory. Everything a tile publishes depends on that
// load (a descriptor on the number, a group sum on the count, by its address), so
// the last tile's CTA, which has then seen every tile, can advance both.
//
// Measured on GB300, graph replay, inputs from HBM, u32, against two levels in turn
// (the last tile of a group reads the group's descriptors and publishes their sum, which
// the tiles of later groups read): 2^17 3.3 -> 2.9 us, 2^18 3.6 -> 3.2, 2^20 5.0 -> 4.3, 2^22
// 8.4 -> 7.9, 2^23 15.3 -> 14.1; u64 2^19 5.4 -> 4.75, 3.5 M 14.3 -> 13.6. With the in-group read
// in a warp of its own beside those of the groups: 2^20 4.3, but 2^22 8.4, 2^23 15.0.
// A flat lookback, in which every tile reads its predecessors' descriptors directly, was
// slower from 2^19 elements on: the reads, quadratic in the tile count, queue on the L2
// lines that hold the descriptors.
constexpr uint32_t kGroupTiles = 32;
constexpr uint32_t kGroupWarps = kMidSums / 32;
constexpr uint64_t kOneTile = 1ull << 40;
static_assert(kGroupTiles * kMidSums == kMidMaxTiles, "one sum per group");

template <typename T>
struct LookbackSmem {
    T part[kGroupWarps];  // what each polling warp has found
    uint32_t used;        // launches that have used the group sums: even ones use one set, odd ones the other
    uint32_t timeout;     // a wait ran past its budget
};

// By all threads; warp 0's get {launch number, launches that have used the group sums}.
__device__ __forceinline__ ptx::u64x2 mid_launch_state(const ScanArgs& a) {
    return threadIdx.x < 32 ? ptx::ld_relaxed_b128(reinterpret_cast<const ptx::u64x2*>(a.mid_launch))
                            : ptx::u64x2{0, 0};
}

// Polls until `done` holds for every lane of the warp, calling look() each
// time; false once the wait budget has run out.
template <class Look>
__device__ __forceinline__ bool mid_poll(const ScanArgs& a, uint32_t lane, Look look) {
    uint32_t polls = 0, backoff = 32;
    uint64_t deadline = 0;
    while (!__all_sync(kFullMask, look())) {
        ++polls;
        if ((polls & 15u) == 1u) {
            bool expired = false;
            if (lane == 0) {
                const uint64_t now = ptx::global_timer_ns();
                if (deadline == 0) deadline = now + a.wait_budget_ns;
                expired = now > deadline || ld_volatile_u32(&a.hdr->error_flags) != 0;
            }
            if (__shfl_sync(kFullMask, expired, 0)) return false;
        }
        if (polls > 64) {
            __nanosleep(backoff);
            backoff = backoff < 1024 ? backoff * 2 : 1024;
        }
    }
    return true;
}

template <typename T, bool GROUPS>
__device__ __forceinline__ char* mid_sums(const ScanArgs& a, const LookbackSmem<T>& sm) {
    return GROUPS ? static_cast<char*>(a.group_desc) + (sm.used & 1u) * (kMidSums * 128u) : nullptr;
}

// By thread 0: publishes tile t's sum `own` (tile 0's with the carry).
// GROUPS = false: a launch of one group.
template <typename T, bool GROUPS>
__device__ __forceinline__ void mid_publish(const ScanArgs& a, uint32_t t, uint64_t tag, T total,
                                            const LookbackSmem<T>& sm) {
    if (t == a.num_tiles - 1) return;
    const uint64_t own = static_cast<uint64_t>(total);
    const uint32_t g = t / kGroupTiles;
    if (t % kGroupTiles != kGroupTiles - 1)
        ptx::st_relaxed_b128(static_cast<ptx::u64x2*>(a.desc) + t * a.desc_stride, MidDesc::pack(kAggregate, tag, own));
    if (GROUPS && (g + 1) * kGroupTiles < a.num_tiles) {
        uint64_t* s = reinterpret_cast<uint64_t*>(mid_sums<T, GROUPS>(a, sm) + g * 128u);
        ptx::red_add_u64(s, kOneTile + static_cast<uint32_t>(own));
        if (sizeof(T) == 8) ptx::red_add_u64(s + 1, kOneTile + (own >> 32));
    }
}

// Returns the sum of the tiles before t, of a launch of more than one, to every
// thread, after its own has been published; sm.timeout is set if a wait ran out.
// `tag` is known to warp 0; sm.used and a cleared sm.timeout are there already.
template <typename T, bool GROUPS>
__device__ __forceinline__ T mid_tile_prefix(const ScanArgs& a, uint32_t t, uint64_t tag, LookbackSmem<T>& sm) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t g = t / kGroupTiles, i = t % kGroupTiles;
    const bool last = t == a.num_tiles - 1;
    const char* sums = mid_sums<T, GROUPS>(a, sm);
    if (warp == 0 || (GROUPS && warp * 32 < g)) {
        const ptx::u64x2* desc = static_cast<const ptx::u64x2*>(a.desc);
        T x = 0;
        bool tile_in = warp != 0 || lane >= i, group_in = !GROUPS || tid >= g;
        const bool ok = mid_poll(a, lane, [&]() {
            // Both loads are issued before the first is looked at.
            ptx::u64x2 w{0, 0}, v{0, 0};
            if (!tile_in) w = ptx::ld_relaxed_b128(desc + (t - i + lane) * a.desc_stride);
            if (!group_in) {
                if (sizeof(T) == 8)
                    v = ptx::ld_relaxed_b128(reinterpret_cast<const ptx::u64x2*>(sums + tid * 128u));
                else
                    v.lo = ptx::ld_relaxed_u64(reinterpret_cast<const uint64_t*>(sums + tid * 128u));
            }
            if (!tile_in && MidDesc::status(w, tag) != kNotReady) {
                tile_in = true;
                x += static_cast<T>(w.lo);
            }
            if (!group_in && v.lo >= kGroupTiles * kOneTile && (sizeof(T) == 4 || v.hi >= kGroupTiles * kOneTile)) {
                group_in = true;
                x += static_cast<T>(v.lo & (kOneTile - 1)) + (sizeof(T) == 8 ? static_cast<T>(v.hi << 32) : T(0));
            }
            return tile_in && group_in;
        });
        x = warp_sum(x);
        if (lane == 0) {
            sm.part[warp] = x;
            if (!ok) sm.timeout = 1u;
        }
    }
    // The other set is used next: by the launch after this one.
    if (GROUPS && t == 0 && tid >= kRowThreads - kMidSums) {
        char* other = static_cast<char*>(a.group_desc) + ((sm.used & 1u) ^ 1u) * (kMidSums * 128u);
        *reinterpret_cast<ptx::u64x2*>(other + (tid - (kRowThreads - kMidSums)) * 128u) = ptx::u64x2{0, 0};
    }
    __syncthreads();
    if (sm.timeout != 0) {
        if (tid == 0) raise_error(a.hdr, kErrLookbackTimeout);
        return T(0);
    }
    T pre = sm.part[0];
#pragma unroll
    for (uint32_t w = 1; w < kGroupWarps; ++w)
        if (GROUPS && w * 32 < g) pre += sm.part[w];
    if (last && tid == 0) {
        ptx::st_relaxed_u64(a.mid_launch, tag + 1);
        if (GROUPS) ptx::st_relaxed_u32(reinterpret_cast<uint32_t*>(a.mid_launch + 1), sm.used + 1);
    }
    return pre;
}

}  // namespace gps
