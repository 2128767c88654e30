// Single-pass chained scan for mid-size inputs: one 16 KB tile per CTA.
//
// The persistent L2-buffered kernel (scan_l2.cuh) pays a pipeline latency of
// about 10 us per launch (unit claim, HBM load, reduce, lookback, reload from
// L2, scan, store), which dominates at small sizes. Here every tile gets its
// own CTA of 256 threads, as in the reference's single-pass kernel
// (ChainedScanDecoupledLookback.cuh:79-139):
//   1. the tile id is the block index: a CTA waits only on lower block
//      indices, which the hardware dispatches first (CUB's decoupled
//      lookback relies on the same order); every wait is bounded, so a
//      violation would surface as GPS_ERR_TIMEOUT, never as a hang;
//   2. load the tile and block-scan it;
//   3. publish the tile's sum and look back: over the tiles of its group of 32
//      and over the sums of the earlier groups, at the same time;
//   4. add the prefix, store.
// The kernels keep their descriptors in a region of the plan of their own,
// tagged with the launch's number, which every CTA reads from the plan's
// header beside its data loads. A descriptor counts only when its tag is the
// current launch's, so a launch needs no clearing memset. The last tile's CTA
// advances the number once its own prefix is known: that prefix rests on
// what every tile before it has published, each by a CTA that had read the
// number, so no CTA of this launch can still be about to read it. No fence is
// on any CTA's path. (A number from the driver will not do:
// %gridid is fixed when a graph is instantiated, the same for all its
// replays.)
#include "gps_device.cuh"
#include "gps_internal.h"
#include "launch_util.h"
#include "tile_rows.cuh"

namespace gps {
namespace {

constexpr int kMidThreads = kRowThreads;
// Resident CTAs per SM of the form that does not hold its tile in registers
// (32 registers a thread).
constexpr int kMidCtasPerSm = 8;

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
// Warp 0 hands that count to the CTA through shared memory, so that it has been
// read before the CTA publishes anything, and the last tile's CTA, which has
// then seen every tile, advances it.
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
    uint32_t set;             // which set of group sums this launch uses
    uint32_t timeout;         // a wait ran past its budget
};

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

// Publishes tile t's sum `total`, known to every thread, and returns the
// prefix before it (with carry_in) to every thread. sm.set and a cleared
// sm.timeout are there already; `tag` is known to warp 0, `used` (the launches
// that have used the group sums) to thread 0. GROUPS = false: one group.
template <typename T, bool GROUPS>
__device__ __forceinline__ T mid_tile_prefix(const ScanArgs& a, uint32_t t, uint64_t tag, uint64_t used, T total,
                                             LookbackSmem<T>& sm) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t g = t / kGroupTiles, i = t % kGroupTiles;
    const bool last = t == a.num_tiles - 1;
    T carry = 0;
    if (a.carry_in != nullptr && t == 0) carry = *static_cast<const T*>(a.carry_in);
    if (a.num_tiles == 1) {
        if (tid == 0 && a.carry_out != nullptr) *static_cast<T*>(a.carry_out) = carry + total;
        return carry;
    }
    char* sums = GROUPS ? static_cast<char*>(a.group_desc) + sm.set * (kMidSums * 128u) : nullptr;
    if (warp == 0 || (GROUPS && warp * 32 < g)) {
        ptx::u64x2* desc = static_cast<ptx::u64x2*>(a.desc);
        if (tid == 0 && !last) {
            const uint64_t own = static_cast<uint64_t>(static_cast<T>(carry + total));
            if (i != kGroupTiles - 1)
                ptx::st_relaxed_b128(desc + t * a.desc_stride, MidDesc::pack(kAggregate, tag, own));
            if (GROUPS && (g + 1) * kGroupTiles < a.num_tiles) {
                uint64_t* s = reinterpret_cast<uint64_t*>(sums + g * 128u);
                ptx::red_add_u64(s, kOneTile + static_cast<uint32_t>(own));
                if (sizeof(T) == 8) ptx::red_add_u64(s + 1, kOneTile + (own >> 32));
            }
        }
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
    if (GROUPS && t == 0 && tid >= kMidThreads - kMidSums) {
        char* other = static_cast<char*>(a.group_desc) + (1u - sm.set) * (kMidSums * 128u);
        *reinterpret_cast<ptx::u64x2*>(other + (tid - (kMidThreads - kMidSums)) * 128u) = ptx::u64x2{0, 0};
    }
    __syncthreads();
    if (sm.timeout != 0) {
        if (tid == 0) raise_error(a.hdr, kErrLookbackTimeout);
        return T(0);
    }
    T pre = carry + sm.part[0];
#pragma unroll
    for (uint32_t w = 1; w < kGroupWarps; ++w)
        if (GROUPS && w * 32 < g) pre += sm.part[w];
    if (last && tid == 0) {
        ptx::st_relaxed_u64(a.mid_launch, tag + 1);
        if (GROUPS) ptx::st_relaxed_u64(&a.hdr->sums_launch, used + 1);
        if (a.carry_out != nullptr) *static_cast<T*>(a.carry_out) = pre + total;
    }
    return pre;
}

// The scan itself. The tile is four rows of 256
// 16-byte chunks, and thread tid holds chunk tid of every row, so each warp
// load or store instruction covers 512 contiguous bytes. The exclusive prefix
// of chunk (r, tid) within the tile is the sum of the rows before r plus the
// chunks of row r before tid: the four chunk sums are warp-scanned together,
// the warp totals go through shared memory in row-major order (row r, warp
// w at r * 8 + w), and one warp scan of those 32 totals gives every (row,
// warp) its offset -- one barrier for the whole block scan; the chunk offsets
// wait in shared memory during the lookback. HELD keeps the tile in registers
// across the lookback, and is the CTAs per SM it is compiled for: four (64
// registers) or six (40). With 0 its chunks are
// read again after it (from L1 or L2): 32 registers, eight CTAs per SM, so that
// up to 1216 tiles (2^22 u32 elements fit on 152 SMs) run in one wave. Which is
// faster turns on the number of waves: up to one wave of the HELD form it is
// ahead (graph replay, u32: 1000 elements 1.43 against 1.62 us, 2^16 2.74 / 2.91,
// 2^20 5.67 / 5.92, 2^21 7.1 / 7.4), beyond it the other (2^22 11.0 / 9.7, 2^23
// 17.8 / 16.7; with four CTAs instead of six, 500 tiles 6.7 / 7.1). There is no shared-memory staging and no mbarrier to set up, so
// every CTA issues its loads as soon as it starts.
//
// ALIGNED = false takes buffers at any element offset from a 16-byte boundary
// (tile_rows.cuh), one row at a time after the lookback, which keeps it at 32
// registers.
// Bound by the same latency chain as the aligned form. Measured on GB300,
// 10,000,019 u32 from a view one element past a boundary, into an aligned
// output: 21.3 us a call, where per-thread element loads and stores (64
// bytes apart across a warp) took 70.9; the generic kernel, which is ahead from
// about there on, 20.2.
//
// GROUPS = false is for launches of one group of tiles, where the code for the
// group sums costs fetches though it is not run (32 captured scans of 2^16 with it
// 84-92 us, without 72-84, by where the plan's memory lies).
template <typename T, bool INCL, bool ALIGNED, int HELD, bool GROUPS>
__global__ void __launch_bounds__(kMidThreads, HELD ? HELD : kMidCtasPerSm) mid_vec_kernel(const ScanArgs a) {
    using Rows = TileRows<T, ALIGNED>;
    constexpr int EPC = Rows::kEpc;
    constexpr int ROWS = Rows::kRows;
    constexpr int WARPS = kMidThreads / 32;
    static_assert(ROWS * WARPS == 32, "one warp scans all (row, warp) totals");
    __shared__ T s_tot[ROWS * WARPS];
    __shared__ T s_off[ROWS][kMidThreads];  // chunk offsets, kept here across the lookback
    __shared__ LookbackSmem<T> lsm;

    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const uint32_t t = blockIdx.x;
    // The tile comes into L2 while the kernel ahead drains. Measured on GB300 (graph
    // replay, inputs from HBM): u32 2^16 2.68 -> 2.56 us, 2^20 5.55 -> 4.98, 2^22 9.7 -> 8.4,
    // 2^23 16.6 -> 15.3 (with the tile of the second wave as well 15.9).
    ptx::prefetch_tile_l2(a.in, t, a.n * sizeof(T), tid);
    ptx::grid_dep_launch();
    ptx::grid_dep_wait();
    // Only warp 0 uses the launch number; its load overlaps the tile's.
    const uint64_t tag = threadIdx.x < 32 ? ptx::ld_relaxed_u64(a.mid_launch) : 0;
    const uint64_t used = GROUPS && threadIdx.x == 0 ? ptx::ld_relaxed_u64(&a.hdr->sums_launch) : 0;
    const Rows rows(a.in, a.out, a.n, t, tid);
    constexpr PlainAccess access;

    T cs[ROWS];
    Chunk<T> held[HELD ? ROWS : 1];
    {
        Chunk<T> q[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) q[r] = rows.load(r, access);
        if constexpr (HELD != 0) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) held[r] = q[r];
        }
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            T x = 0;
#pragma unroll
            for (int e = 0; e < EPC; ++e) x += q[r].v[e];
            cs[r] = x;
        }
    }
    // Block scan of the four rows at once; each thread's four chunk offsets
    // wait in shared memory during the lookback.
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        T wt;
        cs[r] = gps_device::warp_exclusive_scan<gps_device::WarpAlgo::KoggeStone>(cs[r], gps_device::Plus(), &wt);
        if (lane == 0) s_tot[r * WARPS + warp] = wt;
    }
    if (tid == 0) {
        if (GROUPS) lsm.set = static_cast<uint32_t>(used & 1u);
        lsm.timeout = 0u;
    }
    __syncthreads();
    T total;
    {
        const T x = s_tot[lane];
        const T xi = gps_device::warp_inclusive_scan<gps_device::WarpAlgo::KoggeStone>(x, gps_device::Plus());
        const T xe = xi - x;
        total = __shfl_sync(kFullMask, xi, 31);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) s_off[r][tid] = cs[r] + __shfl_sync(kFullMask, xe, r * WARPS + warp);
    }

    const T base = mid_tile_prefix<T, GROUPS>(a, t, tag, used, total, lsm);

    auto scan_chunk = [&](int r, Chunk<T>& q) {
        T acc = base + s_off[r][tid];
#pragma unroll
        for (int e = 0; e < EPC; ++e) {
            const T x = q.v[e];
            if (INCL) {
                acc += x;
                q.v[e] = acc;
            } else {
                q.v[e] = acc;
                acc += x;
            }
        }
    };
    if constexpr (HELD != 0) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            scan_chunk(r, held[r]);
            rows.store(r, held[r], lane, access);
        }
    } else if constexpr (ALIGNED) {
        Chunk<T> q[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) q[r] = rows.load(r, access);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            scan_chunk(r, q[r]);
            rows.store(r, q[r], lane, access);
        }
    } else {
#pragma unroll 1
        for (int r = 0; r < ROWS; ++r) {
            Chunk<T> q = rows.load(r, access);
            scan_chunk(r, q);
            rows.store(r, q, lane, access);
        }
    }
}

template <typename T, bool INCL, bool ALIGNED>
cudaError_t launch_mid_v(const ScanArgs& a0, int num_sms, cudaStream_t stream, LaunchInfo* info) {
    using Rows = TileRows<T, ALIGNED>;
    ScanArgs a = a0;
    // Scans of more tiles than there are group sums for run in pieces, each with
    // the sum through the piece before as its carry.
    char* carries = static_cast<char*>(a0.group_desc) + 2 * 128 * kMidSums;
    if (info) *info = LaunchInfo{static_cast<int>(Rows::tiles(a0.in, a0.n)), kMidThreads, 0};
    for (uint64_t done = 0, piece = 0; done < a0.n; done += a.n, ++piece) {
        a.in = static_cast<const T*>(a0.in) + done;
        a.out = static_cast<T*>(a0.out) + done;
        const uint64_t most = static_cast<uint64_t>(kMidMaxTiles) * Rows::kTile - Rows::lead_of(a.in);
        a.n = a0.n - done < most ? a0.n - done : most;
        a.carry_in = piece == 0 ? a0.carry_in : carries + (piece & 1) * 16;
        a.carry_out = done + a.n == a0.n ? a0.carry_out : carries + ((piece + 1) & 1) * 16;
        a.num_tiles = Rows::tiles(a.in, a.n);
        a.desc_stride = a.num_tiles > kGroupTiles ? kMidDescStride : 1u;
        const int grid = static_cast<int>(a.num_tiles);
        // A dependent launch sets its CTAs up while the kernel ahead finishes: a
        // program that scans one small array after another waits for one launch
        // less each time (2^20 u32: 6.3 -> 5.5 us a call, 32 captured scans of 2^16:
        // 102 -> 89 us).
        // The forms that hold their tile, while the launch is one wave of them.
        const cudaError_t err =
            a.num_tiles <= kGroupTiles
                ? launch_dependent(mid_vec_kernel<T, INCL, ALIGNED, 4, false>, grid, kMidThreads, 0, stream, a)
            : a.num_tiles <= static_cast<uint32_t>(4 * num_sms)
                ? launch_dependent(mid_vec_kernel<T, INCL, ALIGNED, 4, true>, grid, kMidThreads, 0, stream, a)
            : a.num_tiles <= static_cast<uint32_t>(6 * num_sms)
                ? launch_dependent(mid_vec_kernel<T, INCL, ALIGNED, 6, true>, grid, kMidThreads, 0, stream, a)
                : launch_dependent(mid_vec_kernel<T, INCL, ALIGNED, 0, true>, grid, kMidThreads, 0, stream, a);
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

template <typename T, bool INCL>
cudaError_t launch_mid_t(const ScanArgs& a, int num_sms, cudaStream_t stream, LaunchInfo* info) {
    if (((reinterpret_cast<uintptr_t>(a.desc) | reinterpret_cast<uintptr_t>(a.group_desc)) & 15u) != 0 ||
        a.desc == nullptr || a.group_desc == nullptr)
        return cudaErrorInvalidValue;
    const bool aligned = ((reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.out)) & 15u) == 0;
    return aligned ? launch_mid_v<T, INCL, true>(a, num_sms, stream, info)
                   : launch_mid_v<T, INCL, false>(a, num_sms, stream, info);
}

}  // namespace

cudaError_t launch_mid(gps_dtype dtype, bool inclusive, const ScanArgs& a, int num_sms, cudaStream_t stream,
                       LaunchInfo* info) {
    if (dtype == GPS_DTYPE_U64)
        return inclusive ? launch_mid_t<uint64_t, true>(a, num_sms, stream, info)
                         : launch_mid_t<uint64_t, false>(a, num_sms, stream, info);
    return inclusive ? launch_mid_t<uint32_t, true>(a, num_sms, stream, info)
                         : launch_mid_t<uint32_t, false>(a, num_sms, stream, info);
}

}  // namespace gps
