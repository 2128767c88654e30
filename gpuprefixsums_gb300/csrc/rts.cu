// Reduce-then-scan for u32 and u64, without inter-CTA waits, as in the
// reference's ReduceThenScanDispatcher::DispatchKernels{Ex,In}clusive
// (GPUPrefixSumsCUDA/ReduceThenScanDispatcher.cuh:165-187): reduce sums the
// ranges of the input (ReduceThenScan::Reduce, ReduceThenScan.cuh:15-53), the
// sums are scanned (ReduceThenScan::SpineScan, :56-104), propagate scans each
// range from the prefix before it (ReduceThenScan::Propagate, :106-161).
//
// Read from HBM twice, the input alone would cost a half more than the
// single-pass scan. Here it is cut into chunks that stay in L2 (129 MB)
// between the two readings, and every launch but the first and last does the
// reduce of one chunk and the propagate of the chunk before:
//   launch 0      reduce chunk 0
//   launch j      reduce chunk j, then propagate chunk j - 1
//   launch K      propagate chunk K - 1
// A chunk is one range of kRtsTiles 16 KB tiles for every resident CTA, so a
// launch is one even wave. The spine is too short for a launch of its own:
// each propagate CTA adds up the sums of the ranges before its own (at most
// 3 a thread). The launches are dependent launches: a CTA reduces its range
// of chunk j, which rests on no launch before, while the last CTAs of launch
// j - 1 still propagate, and only then waits for that launch to finish.
// Range sums and chunk prefixes therefore have three buffers each: launch
// j + 1 writes while launch j reads, and launch j - 1 has finished by then.
//
// Bound by HBM (25 MB read and 25 written a launch, 7.5 us at the copy rate) and
// the end of each launch: 8.8 us a launch. While the launch ahead drains, no
// output can be written: the last tile of the range to reduce is therefore asked
// for only then, into shared memory, and added at the end (2^28 u32 421 -> 384 us;
// all of the range that way 422; one chunk more between the two readings, without
// the wait, 569). Measured on GB300, u32, against three launches over the whole
// input (reduce, a one-CTA spine over one sum a tile, propagate): 2^20 9.5 -> 5.1
// us, 2^24 39 -> 31, 2^26 142 -> 102, 2^28 542 -> 384; a view of 10,000,019 elements
// off a 16-byte boundary 167 -> 25.
#include "launch_util.h"
#include "tile_rows.cuh"

namespace gps {

namespace {

constexpr int kRtsCtasPerSm = 5;
// Tiles of a CTA's range in one chunk, at most: 25 MB a chunk. Two chunks wait
// in L2 at a time, next to what is being written. Measured on GB300, 2^28 u32:
// 2 tiles 384 us, 3 tiles 419 and 4 459 (part of the chunk has left L2 by the
// second reading), 1 tile 516 before the late tile (the end of a launch costs 2
// us); 4 or 6 CTAs per SM 393 and 387. Without evict-last loads in the reduce 491
// against 421.
constexpr uint32_t kRtsTiles = 2;

struct RtsArgs {
    const void* in;
    void* out;
    uint64_t n;
    uint32_t tiles;
    uint32_t range_tiles;  // tiles per range; a chunk is gridDim.x ranges
    uint32_t chunk;        // this launch reduces it and propagates the one before
    uint32_t chunks;
    void* sums;      // [3][gridDim.x] range sums
    void* prefixes;  // [3] sum of the chunks before
    const void* carry_in;
    void* carry_out;
    WsHeader* hdr;
    uint64_t wait_budget_ns;
};

template <typename T, bool INCL, bool ALIGNED>
__global__ void __launch_bounds__(kRowThreads, kRtsCtasPerSm) rts_kernel(const RtsArgs a) {
    using Rows = TileRows<T, ALIGNED>;
    constexpr int ROWS = Rows::kRows;
    constexpr int WARPS = kRowThreads / 32;
    static_assert(ROWS * WARPS == 32, "one warp scans all (row, warp) totals");
    __shared__ T s_tot[2][32];
    __shared__ T s_pre[2][WARPS];
    __shared__ uint64_t s_bar;
    extern __shared__ __align__(128) uint8_t s_raw[];  // one tile, where a launch has a reduce and a propagate part
    T* s_stage = reinterpret_cast<T*>(s_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t ranges = gridDim.x, b = blockIdx.x;
    T* sums = static_cast<T*>(a.sums);
    T* prefixes = static_cast<T*>(a.prefixes);

    if (a.chunk == 0) {
        // The range comes into L2 while the kernel ahead drains (2^24 u32 31.0 -> 29.4 us).
        for (uint32_t k = 0; k < a.range_tiles; ++k)
            ptx::prefetch_tile_l2(a.in, b * a.range_tiles + k, a.n * sizeof(T), tid);
        ptx::grid_dep_wait();  // the input's producers
    }
    // Reduce: one range of chunk a.chunk. L2 keeps what it reads. The last tile
    // of the range is only asked for before the wait below, into shared memory,
    // and added at the end: it keeps HBM busy while the launch ahead drains.
    const uint64_t r_begin = (static_cast<uint64_t>(a.chunk) * ranges + b) * a.range_tiles;
    uint64_t r_end = a.chunk < a.chunks ? min(r_begin + a.range_tiles, static_cast<uint64_t>(a.tiles)) : 0;
    bool deferred = false;
    if (a.chunk != 0 && r_begin < r_end) {
        const Rows rows(a.in, a.out, a.n, static_cast<uint32_t>(r_end - 1), 0);
        deferred = rows.full;
        if (deferred) {
            --r_end;
            if (tid == 0) {
                ptx::mbar_init(&s_bar, 1);
                ptx::fence_mbar_init();
            }
        }
    }
    T acc = 0;
    auto publish_sum = [&]() {
        acc = warp_sum(acc);
        __syncthreads();
        if (lane == 0) s_pre[0][warp] = acc;
        __syncthreads();
        if (tid == 0) {
            T x = 0;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) x += s_pre[0][w];
            sums[(a.chunk % 3) * ranges + b] = x;
        }
    };
    if (a.chunk < a.chunks) {
        const PolicyAccess pol{ptx::policy_evict_last()};
#pragma unroll 2
        for (uint64_t t = r_begin; t < r_end; ++t) {
            const Rows rows(a.in, a.out, a.n, static_cast<uint32_t>(t), tid);
            Chunk<T> q[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) q[r] = rows.load(r, pol);
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
#pragma unroll
                for (int e = 0; e < Rows::kEpc; ++e) acc += q[r].v[e];
        }
        if (!deferred) publish_sum();
        __syncthreads();
    }
    if (a.chunk == 0) {
        ptx::grid_dep_launch();
        return;
    }

    // Propagate: the same range of the chunk before. Its first tile is loaded
    // and scanned before the wait, which only guards the range sums.
    const uint32_t c = a.chunk - 1;
    const PolicyAccess pol{ptx::policy_evict_first()};
    const uint64_t begin = (static_cast<uint64_t>(c) * ranges + b) * a.range_tiles;
    const uint64_t end = min(begin + a.range_tiles, static_cast<uint64_t>(a.tiles));
    T pre = 0;
    for (uint64_t t = begin; t < end || t == begin; ++t) {
        const bool live = t < end;  // a range past the end still takes part in the barriers
        const Rows rows(a.in, a.out, a.n, static_cast<uint32_t>(live ? t : 0), tid);
        Chunk<T> q[ROWS] = {};
        if (live) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) q[r] = rows.load(r, pol);
        }
        T off[ROWS];
        T* tot = s_tot[t & 1u];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            T x = 0;
#pragma unroll
            for (int e = 0; e < Rows::kEpc; ++e) x += q[r].v[e];
            const T inc = warp_inclusive_scan(x, lane);
            if (lane == 31) tot[r * WARPS + warp] = inc;
            off[r] = inc - x;
        }
        if (t == begin) {
            if (deferred && tid == 0) {
                const Rows last(a.in, a.out, a.n, static_cast<uint32_t>(r_end), 0);
                ptx::mbar_arrive_expect_tx(&s_bar, 16384u);
                ptx::bulk_load_hint(s_stage, last.src, 16384u, &s_bar, ptx::policy_evict_last());
            }
            ptx::grid_dep_wait();
            ptx::grid_dep_launch();
            const T* cs = sums + (c % 3) * ranges;
            T mine = 0, all = 0;
            for (uint32_t i = tid; i < ranges; i += kRowThreads) {
                const T x = cs[i];
                mine += i < b ? x : T(0);
                all += x;
            }
            pre = c != 0 ? prefixes[c % 3] : a.carry_in != nullptr ? *static_cast<const T*>(a.carry_in) : T(0);
            mine = warp_sum(mine);
            if (b == 0) all = warp_sum(all);
            if (lane == 0) {
                s_pre[0][warp] = mine;
                s_pre[1][warp] = all;
            }
        }
        __syncthreads();
        if (t == begin) {
            if (b == 0 && tid == 0) {
                T x = pre;
#pragma unroll
                for (int w = 0; w < WARPS; ++w) x += s_pre[1][w];
                prefixes[(c + 1) % 3] = x;
                if (a.chunk == a.chunks && a.carry_out != nullptr) *static_cast<T*>(a.carry_out) = x;
            }
#pragma unroll
            for (int w = 0; w < WARPS; ++w) pre += s_pre[0][w];
        }
        if (!live) break;
        // Every warp scans the 32 (row, warp) totals.
        const T x = tot[lane];
        const T xi = warp_inclusive_scan(x, lane);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            T run = pre + off[r] + __shfl_sync(kFullMask, xi - x, r * WARPS + warp);
#pragma unroll
            for (int e = 0; e < Rows::kEpc; ++e) {
                const T y = q[r].v[e];
                if (INCL) {
                    run += y;
                    q[r].v[e] = run;
                } else {
                    q[r].v[e] = run;
                    run += y;
                }
            }
            rows.store(r, q[r], lane, pol);
        }
        pre += __shfl_sync(kFullMask, xi, 31);
    }
    if (deferred) {
        if (!ptx::mbar_try_wait(&s_bar, 0) &&
            !ptx::mbar_wait_bounded(&s_bar, 0, ptx::global_timer_ns() + a.wait_budget_ns))
            raise_error(a.hdr, kErrPipelineTimeout);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            const Chunk<T> q = reinterpret_cast<const Chunk<T>*>(s_stage)[r * kRowThreads + tid];
#pragma unroll
            for (int e = 0; e < Rows::kEpc; ++e) acc += q.v[e];
        }
        publish_sum();
    }
}

// Ranges per chunk, tiles per range and chunks of a scan of `tiles` tiles:
// the fewest chunks, cut evenly.
struct RtsShape {
    uint32_t ranges, range_tiles, chunks;
};
RtsShape rts_shape(uint32_t tiles, int num_sms) {
    const uint32_t ranges = static_cast<uint32_t>(persistent_grid(tiles, kRtsCtasPerSm, num_sms));
    const uint32_t per_range = (tiles + ranges - 1) / ranges;
    const uint32_t chunks = (per_range + kRtsTiles - 1) / kRtsTiles;
    const uint32_t range_tiles = (per_range + chunks - 1) / chunks;
    return RtsShape{ranges, range_tiles, (per_range + range_tiles - 1) / range_tiles};
}

template <typename T, bool ALIGNED>
cudaError_t dispatch_rts(bool inclusive, const ScanArgs& s, void* scratch, int num_sms, cudaStream_t stream,
                         LaunchInfo* info) {
    const uint32_t tiles = TileRows<T, ALIGNED>::tiles(s.in, s.n);
    const RtsShape sh = rts_shape(tiles, num_sms);
    T* sums = static_cast<T*>(scratch);
    RtsArgs a{s.in,      s.out, s.n,       tiles,
              sh.range_tiles, 0,     sh.chunks, sums,
              sums + 3ull * static_cast<uint64_t>(kRtsCtasPerSm * num_sms), s.carry_in, s.carry_out, s.hdr, s.wait_budget_ns};
    const int grid = static_cast<int>(sh.ranges);
    const size_t smem = sh.chunks > 1 ? 16384 : 0;
    if (info) *info = LaunchInfo{grid, kRowThreads, smem, sh.chunks + 1};
    for (; a.chunk <= sh.chunks; ++a.chunk) {
        const cudaError_t err =
            inclusive ? launch_dependent(rts_kernel<T, true, ALIGNED>, grid, kRowThreads, smem, stream, a)
                      : launch_dependent(rts_kernel<T, false, ALIGNED>, grid, kRowThreads, smem, stream, a);
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

template <typename T>
cudaError_t dispatch_rts(bool inclusive, const ScanArgs& a, void* scratch, int num_sms, cudaStream_t stream,
                         LaunchInfo* info) {
    const bool aligned = ((reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.out)) & 15u) == 0;
    return aligned ? dispatch_rts<T, true>(inclusive, a, scratch, num_sms, stream, info)
                   : dispatch_rts<T, false>(inclusive, a, scratch, num_sms, stream, info);
}

}  // namespace

uint32_t rts_tile_elems(gps_dtype dtype) { return 16384u / static_cast<uint32_t>(dtype_size(dtype)); }

uint64_t rts_scratch_elems(int num_sms) { return 3ull * static_cast<uint64_t>(kRtsCtasPerSm * num_sms) + 3; }

uint32_t rts_launches(uint64_t n, uint32_t tile_elems, int num_sms) {
    return rts_shape(static_cast<uint32_t>((n + tile_elems - 1) / tile_elems), num_sms).chunks + 1;
}

cudaError_t launch_rts(gps_dtype dtype, bool inclusive, const ScanArgs& a, void* scratch, int num_sms,
                       cudaStream_t stream, LaunchInfo* info) {
    if (dtype == GPS_DTYPE_U64) return dispatch_rts<uint64_t>(inclusive, a, scratch, num_sms, stream, info);
    return dispatch_rts<uint32_t>(inclusive, a, scratch, num_sms, stream, info);
}

}  // namespace gps
