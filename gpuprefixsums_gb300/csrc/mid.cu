// Single-pass chained scan for mid-size inputs: one 16 KB tile per CTA.
//
// The persistent kernel of large scans (scan_seg.cuh) pays a pipeline latency of
// 8 to 10 us per launch (unit claim, HBM load, reduce, lookback, reload from
// L2, scan, store), which dominates at small sizes. Here every tile gets its
// own CTA of 256 threads, as in the reference's single-pass kernel
// (ChainedScanDecoupledLookback.cuh:79-139):
//   1. the tile id is the block index: a CTA waits only on lower block
//      indices, which the hardware dispatches first (CUB's decoupled
//      lookback relies on the same order); every wait is bounded, so a
//      violation would surface as GPS_ERR_TIMEOUT, never as a hang;
//   2. load the tile and block-scan it;
//   3. publish the tile's sum and look back (mid_lookback.cuh): over the tiles of its group of 32
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
#include "mid_lookback.cuh"

namespace gps {
namespace {

constexpr int kMidThreads = kRowThreads;
// Resident CTAs per SM of the form that does not hold its tile in registers
// (32 registers a thread).
constexpr int kMidCtasPerSm = 8;

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
// fastest turns on the number of waves: the form that holds most while the launch
// is one wave of it. Measured on GB300 (graph replay, inputs from HBM, us, HELD 4 / 6 /
// 0): u32 256 tiles 4.36 / 4.49 / 4.66, 608 tiles 5.64 / 6.04 / 6.08, 700 tiles 8.22 / 6.23 / 6.79,
// 912 tiles 9.32 / 7.14 / 7.73, 1024 tiles 9.84 / 9.31 / 8.27, 1216 tiles 10.9 / 10.5 / 9.6; u64 and views
// alike. There is no shared-memory staging and no mbarrier to set up, so
// every CTA issues its loads as soon as it starts.
//
// ALIGNED = false takes buffers at any element offset from a 16-byte boundary
// (tile_rows.cuh), one row at a time after the lookback, which keeps it at 32
// registers.
// Bound by the same latency chain as the aligned form. Measured on GB300,
// 10,000,019 u32 from a view one element past a boundary, into an aligned
// output: 20.0 us a call, where per-thread element loads and stores (64
// bytes apart across a warp) took 70.9; 1024 tiles 9.5 us against 8.3 aligned. The
// generic kernel is ahead from 2420 tiles on (mid_max_bytes()).
//
// GROUPS = false is for launches of one group of tiles, where the code for the
// group sums costs fetches though it is not run (32 captured scans of 2^16 with it
// 84-92 us, without 72-84, by where the plan's memory lies; 78-86 in the latest
// measurement, over eight plans of one process).
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
    const ptx::u64x2 launch = mid_launch_state(a);
    const uint64_t tag = launch.lo;
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
        if (GROUPS) lsm.used = static_cast<uint32_t>(launch.hi);
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

    T carry = 0;  // of tile 0; the others' is in its sum
    if (a.carry_in != nullptr && t == 0) carry = *static_cast<const T*>(a.carry_in);
    T base = carry;
    if (a.num_tiles > 1) {
        if (tid == 0) mid_publish<T, GROUPS>(a, t, tag, carry + total, lsm);
        base += mid_tile_prefix<T, GROUPS>(a, t, tag, lsm);
    }
    if (a.carry_out != nullptr && tid == 0 && t == a.num_tiles - 1) *static_cast<T*>(a.carry_out) = base + total;

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
    if (info) *info = LaunchInfo{static_cast<int>(Rows::tiles(a0.in, a0.n)), kMidThreads, 0, 0};
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
        if (info) ++info->launches;
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
