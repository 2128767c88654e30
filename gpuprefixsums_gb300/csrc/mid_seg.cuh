// One 16 KB tile per CTA for any scan operation of scan_ops.cuh, plain or
// segmented: the small and mid sizes of the generic kernel (scan_seg.cuh),
// whose pipeline (unit claim, prefetch, reduce pass, aggregator, lookback,
// second load, scan pass, retirement) has a latency of 8 to 10 us.
//
// Structure of a CTA (256 threads, tile id = block index, as in mid.cu: a CTA
// waits on lower block indices only, and every wait is bounded):
//   1. load the tile, 16-byte chunks coalesced over the warp, into shared
//      memory; thread i owns the 64 contiguous bytes of chunks 4i .. 4i + 3.
//      Chunk c sits at c ^ ((c >> 3) & 3), so that both the coalesced stores
//      and each thread's own reads touch every bank once;
//   2. segmented: while the loads are in flight, find the first offset of the
//      tile, with 256 probes a round until 1024 are left, and mark the heads in
//      a bitmap;
//   3. aggregate each thread's items, scan over the block, publish the tile's
//      aggregate;
//   4. lookback in a fixed order (below);
//   5. scan the items from shared memory, store coalesced.
// The tile is read from HBM once and waits in shared memory. Latency bounds
// it: one HBM read, two L2 round trips (in-group, groups), a store.
//
// Fixed-order lookback: tiles form groups of kMidSegGroup. A tile's
// descriptor only ever holds its aggregate, and the last tile of a group
// publishes the group's aggregate once it has read its in-group predecessors.
// The prefix of a tile is fold(aggregates of the groups before) . fold(
// aggregates of the group's tiles before it), each fold of one fixed shape
// (every lane its consecutive entries in order, then an order-keeping
// butterfly). No value depends on timing, so floating-point results repeat
// bit for bit, and no prefix passes from tile to tile or group to group: all
// tiles wait for the same two L2 round trips instead of a chain.
//
// Measured on GB300, graph replay, inputs from HBM, against the generic kernel
// in units of 4 tiles: FP32 2^20 5.2 against 8.4 us, 2^22 9.4 / 12.5; compensated
// FP32 2^20 6.6 / 9.2, 2^22 11.9 / 13.8; batched u32 (500 segments) 2^20 5.3 / 10.3;
// 300,000 segments in 2^20 elements 6.7 / 17.2; 500 compensated segments of 2.2 M
// 8.4 / 14.7. Groups of 64 tiles against 32 / 128: FP32 2^20 5.16 / 5.33 / 5.33 us, compensated
// 2^22 11.9 / 12.5 / 12.5.
#pragma once
#include "scan_seg.cuh"
#include "segment_search.h"

namespace gps {

constexpr int kMidSegThreads = 256;

// 16-byte descriptor words, as many as the chain value has 64-bit words:
//   lo: value bits; hi: status:1 (bit 63) | head flag:1 (bit 62) | launch
//   number:62.
// The launch number comes from the plan's header, which the last tile's CTA
// advances once every tile has published (see mid.cu): a word of an earlier
// launch never matches, and a launch needs no clearing.
constexpr uint64_t kMidSegTagMask = (1ull << 62) - 1;

template <class Op>
__device__ __forceinline__ void mid_seg_store(ptx::u64x2* d, uint64_t tag, bool flag, typename Op::C c) {
#pragma unroll
    for (int w = 0; w < Op::kDescWords; ++w) {
        ptx::u64x2 x;
        x.lo = Op::chain_word(c, w);
        x.hi = (1ull << 63) | (flag ? 1ull << 62 : 0ull) | (tag & kMidSegTagMask);
        ptx::st_relaxed_b128(d + w, x);
    }
}

// False unless every word of the descriptor carries this launch's number.
template <class Op>
__device__ __forceinline__ bool mid_seg_decode(const ptx::u64x2 (&d)[Op::kDescWords], uint64_t tag, bool& flag,
                                               typename Op::C& c) {
    uint64_t words[Op::kDescWords];
    bool ok = true;
#pragma unroll
    for (int w = 0; w < Op::kDescWords; ++w) {
        const ptx::u64x2 x = d[w];
        ok = ok && (x.hi >> 63) != 0 && (x.hi & kMidSegTagMask) == (tag & kMidSegTagMask);
        flag = ((x.hi >> 62) & 1u) != 0;
        words[w] = x.lo;
    }
    if (ok) c = Op::chain_from_words(words);
    return ok;
}

// Fold, in order, of the `cnt` descriptors from `d` on (stride `ws` words),
// at most 32 * K: lane l takes entries l * K .. l * K + K - 1. Waits until
// all of them are published; false once the wait budget has run out.
template <class Op, int K>
__device__ __forceinline__ bool mid_seg_fold(const ScanArgs& a, const ptx::u64x2* d, uint32_t ws, uint32_t cnt,
                                             uint64_t tag, uint32_t lane, typename Op::C& out, bool& out_flag) {
    using C = typename Op::C;
    C v[K];
    bool f[K];
    uint32_t ready = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        v[j] = Op::chain_zero();
        f[j] = false;
        if (lane * K + j >= cnt) ready |= 1u << j;
    }
    uint32_t polls = 0, backoff = 32;
    uint64_t deadline = 0;
    while (true) {
        // All loads of a poll are issued before the first is looked at.
        ptx::u64x2 x[K][Op::kDescWords];
#pragma unroll
        for (int j = 0; j < K; ++j)
#pragma unroll
            for (int w = 0; w < Op::kDescWords; ++w) {
                x[j][w] = ptx::u64x2{0, 0};
                if (!((ready >> j) & 1u)) x[j][w] = ptx::ld_relaxed_b128(d + static_cast<uint64_t>(lane * K + j) * ws + w);
            }
#pragma unroll
        for (int j = 0; j < K; ++j) {
            bool hf = false;
            C cv;
            if (!((ready >> j) & 1u) && mid_seg_decode<Op>(x[j], tag, hf, cv)) {
                v[j] = cv;
                f[j] = hf;
                ready |= 1u << j;
            }
        }
        if (__all_sync(kFullMask, ready == (1u << K) - 1u)) break;
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
    C c = v[0];
    bool fl = f[0];
#pragma unroll
    for (int j = 1; j < K; ++j) {
        c = f[j] ? v[j] : Op::chain_add(c, v[j]);
        fl = fl || f[j];
    }
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const C oc = Op::chain_shfl_xor(c, m);
        const bool of = __shfl_xor_sync(kFullMask, fl, m) != 0;
        if (lane & static_cast<uint32_t>(m))
            c = fl ? c : Op::chain_add(oc, c);
        else
            c = of ? oc : Op::chain_add(c, oc);
        fl = fl || of;
    }
    out = c;
    out_flag = fl;
    return true;
}

// Run by warp 0 of tile t: publishes the tile's aggregate (and its group's, by
// the group's last tile) and folds the aggregates before it into `pre`. The
// last tile waits for all groups and advances the launch number. False once
// the wait budget has run out.
template <class Op>
__device__ __forceinline__ bool mid_seg_prefix(const ScanArgs& a, uint32_t t, uint64_t tag, typename Op::C agg,
                                               bool flag, uint32_t lane, typename Op::C& pre) {
    using C = typename Op::C;
    constexpr int KT = static_cast<int>(kMidSegGroup / 32);
    constexpr int KG = static_cast<int>((kMidSegMaxTiles / kMidSegGroup + 31) / 32);
    const uint32_t ws = a.desc_stride;
    ptx::u64x2* d1 = static_cast<ptx::u64x2*>(a.desc);
    ptx::u64x2* d2 = static_cast<ptx::u64x2*>(a.group_desc);
    if (lane == 0) mid_seg_store<Op>(d1 + static_cast<uint64_t>(t) * ws, tag, flag, agg);
    const uint32_t g = t / kMidSegGroup;
    const uint32_t i0 = g * kMidSegGroup;
    C in = Op::chain_zero(), gp = Op::chain_zero();
    bool inf = false, gpf = false, ok = true;
    // A launch of up to 32 tiles reads one descriptor a lane.
    if (t != i0) {
        const ptx::u64x2* dg = d1 + static_cast<uint64_t>(i0) * ws;
        ok = a.num_tiles <= 32 ? mid_seg_fold<Op, 1>(a, dg, ws, t - i0, tag, lane, in, inf)
                               : mid_seg_fold<Op, KT>(a, dg, ws, t - i0, tag, lane, in, inf);
    }
    if (ok && lane == 0 && t - i0 == kMidSegGroup - 1)
        mid_seg_store<Op>(d2 + static_cast<uint64_t>(g) * kMidDescStride, tag, inf || flag,
                          flag ? agg : Op::chain_add(in, agg));
    const bool last = t == a.num_tiles - 1;
    if (ok && g != 0 && (!inf || last)) {
        ok = mid_seg_fold<Op, KG>(a, d2, kMidDescStride, g, tag, lane, gp, gpf);
        if (!inf) in = t == i0 ? gp : Op::chain_add(gp, in);
    }
    if (ok && last && lane == 0) ptx::st_relaxed_u64(a.mid_launch, tag + 1);
    pre = in;
    return ok;
}

// CTAS: resident CTAs per SM the kernel is compiled for. Few leave it more
// registers, the faster form while a launch fits one wave of them; larger
// launches want more tiles in flight: the smallest of 4, 6 and 8 that takes the
// launch in one wave (segmented scans at most 6, structs always 4). Measured on
// GB300 (graph replay, inputs from HBM, us, 4 / 6 / 8 CTAs): FP32 256 tiles 5.12 / 5.19 / 5.42, 768
// tiles 9.47 / 7.53 / 8.39, 1024 tiles 11.3 / 10.4 / 9.5; compensated 1024 tiles 14.1 / 13.2 / 11.8;
// batched (4 / 6) compensated 500 tiles 8.27 / 9.46, 768 tiles 12.2 / 10.6; batched u64 500 tiles
// 6.65 / 7.79; select u32 500 tiles 5.11 / 5.07 / 5.78, 608 tiles 5.44 / 5.60 / 5.46, 768 tiles 8.16 / 6.13 /
// 7.00, 1024 tiles 8.94 / 8.90 / 7.85 (1300 tiles, two waves of every form, 10.1 / 9.9 / 11.0).
inline int mid_seg_ctas(uint32_t tiles, int num_sms, int most) {
    for (int c = 4; c < most; c += 2)
        if (tiles <= static_cast<uint32_t>(c * num_sms)) return c;
    return most;
}

template <class Op, bool INCL, bool SEG, int CTAS>
__global__ void __launch_bounds__(kMidSegThreads, CTAS)
    mid_seg_kernel(const ScanArgs a, const SegArgs sg) {
    using T = typename Op::T;
    using S = typename Op::S;
    using C = typename Op::C;
    constexpr int TILE = 16384 / static_cast<int>(sizeof(T));
    constexpr int EPC = 16 / static_cast<int>(sizeof(T));
    constexpr int ITEMS = TILE / kMidSegThreads;  // 64 bytes
    constexpr int CHUNKS = 4;
    constexpr int WARPS = kMidSegThreads / 32;
    constexpr int kHeadWords = TILE / 32;
    static_assert(ITEMS == CHUNKS * EPC, "four chunks a thread");

    __shared__ __align__(16) Chunk<T> s_tile[CHUNKS * kMidSegThreads];
    __shared__ S s_wtot[WARPS];
    __shared__ uint8_t s_wflag[WARPS];
    __shared__ uint32_t s_head[SEG ? kHeadWords : 1];
    __shared__ C s_pre;

    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    const uint32_t warp = tid >> 5;
    const uint32_t t = blockIdx.x;
    // As in mid.cu: FP32 2^20 5.6 -> 5.1 us, 2^22 10.5 -> 9.1; 500 compensated scans 9.8 -> 8.8.
    ptx::prefetch_tile_l2(a.in, t, a.n * sizeof(T), tid);
    ptx::grid_dep_launch();
    ptx::grid_dep_wait();
    const uint64_t tag = threadIdx.x < 32 ? ptx::ld_relaxed_u64(a.mid_launch) : 0;
    const uint64_t t0 = static_cast<uint64_t>(t) * TILE;
    const uint32_t cnt = static_cast<uint32_t>(min(static_cast<uint64_t>(TILE), a.n - t0));
    auto slot = [](uint32_t c) -> uint32_t { return c ^ ((c >> 3) & 3u); };

    // 1. Load.
    const T* src = static_cast<const T*>(a.in) + t0;
    Chunk<T> q[CHUNKS];
#pragma unroll
    for (int r = 0; r < CHUNKS; ++r) {
        const uint32_t off = (r * kMidSegThreads + tid) * EPC;
        if (off + EPC <= cnt) {
            q[r] = *reinterpret_cast<const Chunk<T>*>(src + off);
        } else {
#pragma unroll
            for (int e = 0; e < EPC; ++e) q[r].v[e] = off + e < cnt ? src[off + e] : T{};
        }
    }
    // 2. Segment heads: offsets o with t0 <= o < t0 + cnt.
    if constexpr (SEG) {
        for (uint32_t w = tid; w < kHeadWords; w += kMidSegThreads) s_head[w] = 0u;
        const uint32_t nseg = sg.num_segments;
        // Offsets a thread reads at a time. An interval that one such reading covers is
        // not narrowed further: up to 1024 segments no probe is left, and one latency
        // less ahead of the scan (500 compensated scans 8.8 -> 8.5 us, 1000 segments of
        // 2^20 u32 5.66 -> 5.44; from 5000 segments on no change).
        constexpr uint32_t kBatch = 4;
        OffsetInterval at{0, nseg};
        while (at.size() > kBatch * kMidSegThreads) {
            const uint32_t probe = at.probe(tid, kMidSegThreads);
            const bool below = probe < at.size() && sg.offsets[at.lo + probe] < t0;
            at.narrow(static_cast<uint32_t>(__syncthreads_count(below)), kMidSegThreads);
        }
        __syncthreads();
        for (uint64_t cur = at.lo;; cur += kBatch * kMidSegThreads) {
            uint64_t o[kBatch];
#pragma unroll
            for (uint32_t j = 0; j < kBatch; ++j) {
                const uint64_t idx = cur + j * kMidSegThreads + tid;
                o[j] = idx < nseg ? sg.offsets[idx] : ~0ull;
            }
#pragma unroll
            for (uint32_t j = 0; j < kBatch; ++j) {
                if (o[j] >= t0 && o[j] < t0 + cnt) {
                    const uint32_t pos = static_cast<uint32_t>(o[j] - t0);
                    atomicOr(&s_head[pos >> 5], 1u << (pos & 31u));
                }
            }
            if (__syncthreads_or(o[kBatch - 1] >= t0 + cnt)) break;
        }
    }
#pragma unroll
    for (int r = 0; r < CHUNKS; ++r) s_tile[slot(r * kMidSegThreads + tid)] = q[r];
    __syncthreads();

    // 3. Block scan of the threads' aggregates.
    auto load_items = [&](T(&v)[ITEMS]) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            const Chunk<T> x = s_tile[slot(tid * CHUNKS + c)];
#pragma unroll
            for (int e = 0; e < EPC; ++e) v[c * EPC + e] = x.v[e];
        }
    };
    uint32_t hb = 0;
    if constexpr (SEG) hb = (s_head[tid * ITEMS / 32] >> ((tid * ITEMS) & 31u)) & ((1u << ITEMS) - 1u);
    // Warps without a head take the plain chains (for compensated FP32 the sum is
    // packed; a batch of 500 compensated scans 10.5 -> 9.7 us a call).
    const bool has_heads = SEG && __any_sync(kFullMask, hb != 0u);
    S x;
    bool xf = SEG && hb != 0u;
    {
        T v[ITEMS];
        load_items(v);
        x = has_heads ? thread_aggregate<Op, ITEMS, true>(v, hb) : thread_aggregate<Op, ITEMS, false>(v, 0u);
    }
    warp_scan_incl<Op, SEG>(x, xf, lane);
    if (lane == 31) {
        s_wtot[warp] = x;
        if (SEG) s_wflag[warp] = xf ? 1 : 0;
    }
    S pre = Op::shfl_up(x, 1);
    bool pf = SEG ? __shfl_up_sync(kFullMask, xf, 1) != 0 : false;
    if (lane == 0) {
        pre = Op::zero();
        pf = false;
    }
    __syncthreads();
    S tot = Op::zero();
    bool totf = false;
    {
        S wp = Op::zero();
        bool wpf = false;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            if (static_cast<uint32_t>(w) == warp) {
                wp = tot;
                wpf = totf;
            }
            seg_combine<Op>(tot, totf, s_wtot[w], SEG && s_wflag[w] != 0);
        }
        // The state before this thread within the tile.
        seg_combine<Op>(wp, wpf, pre, pf);
        pre = wp;
        pf = wpf;
    }

    // 4. Publish and look back.
    if (a.num_tiles > 1) {
        if (warp == 0) {
            C before;
            const bool ok = mid_seg_prefix<Op>(a, t, tag, Op::to_chain(Op::norm(tot)), totf, lane, before);
            if (lane == 0) {
                if (!ok) raise_error(a.hdr, kErrLookbackTimeout);
                s_pre = before;
            }
        }
        __syncthreads();
    }
    const S run = a.num_tiles > 1 ? Op::from_chain(s_pre) : Op::zero();
    const S base = pf ? pre : Op::combine(run, pre);

    // 5. Scan and store.
    {
        T v[ITEMS];
        load_items(v);
        // (A second copy of the output chain only pays where the chain is long.)
        if (sizeof(S) > sizeof(T) ? has_heads : SEG)
            thread_outputs<Op, ITEMS, true, INCL>(v, base, hb);
        else
            thread_outputs<Op, ITEMS, false, INCL>(v, base, 0u);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
            Chunk<T> y;
#pragma unroll
            for (int e = 0; e < EPC; ++e) y.v[e] = v[c * EPC + e];
            s_tile[slot(tid * CHUNKS + c)] = y;
        }
    }
    __syncthreads();
    T* dst = static_cast<T*>(a.out) + t0;
#pragma unroll
    for (int r = 0; r < CHUNKS; ++r) {
        const uint32_t off = (r * kMidSegThreads + tid) * EPC;
        const Chunk<T> y = s_tile[slot(r * kMidSegThreads + tid)];
        if (off + EPC <= cnt) {
            *reinterpret_cast<Chunk<T>*>(dst + off) = y;
        } else {
#pragma unroll
            for (int e = 0; e < EPC; ++e)
                if (off + e < cnt) dst[off + e] = y.v[e];
        }
    }
}

template <class Op>
cudaError_t launch_mid_seg(bool inclusive, const ScanArgs& a0, const SegArgs* sg, int num_sms, cudaStream_t stream,
                           LaunchInfo* info) {
    if (((reinterpret_cast<uintptr_t>(a0.desc) | reinterpret_cast<uintptr_t>(a0.group_desc)) & 15u) != 0 ||
        a0.desc == nullptr || a0.group_desc == nullptr || a0.num_tiles > kMidSegMaxTiles)
        return cudaErrorInvalidValue;
    ScanArgs a = a0;
    a.desc_stride = a.num_tiles > 32 ? kMidDescStride : static_cast<uint32_t>(Op::kDescWords);
    const int grid = static_cast<int>(a.num_tiles);
    if (info) *info = LaunchInfo{grid, kMidSegThreads, 0};
    const SegArgs none{nullptr, 0};
    // Dependent launches, as in mid.cu (FP32 2^20: 7.2 -> 5.8 us a call, a batch of
    // 500 compensated scans 12.1 -> 10.5).
    auto launch = [&](void (*kern)(ScanArgs, SegArgs), const SegArgs& s) {
        return launch_dependent(kern, grid, kMidSegThreads, 0, stream, a, s);
    };
    constexpr int kMost = sizeof(typename Op::S) > 8 ? 4 : 8;
    constexpr int k6 = kMost < 6 ? kMost : 6;
    const int ctas = mid_seg_ctas(a.num_tiles, num_sms, sg != nullptr ? k6 : kMost);
    if (sg != nullptr) {
        if (ctas == 4)
            return inclusive ? launch(mid_seg_kernel<Op, true, true, 4>, *sg)
                             : launch(mid_seg_kernel<Op, false, true, 4>, *sg);
        return inclusive ? launch(mid_seg_kernel<Op, true, true, k6>, *sg)
                         : launch(mid_seg_kernel<Op, false, true, k6>, *sg);
    }
    if (ctas == 4)
        return inclusive ? launch(mid_seg_kernel<Op, true, false, 4>, none)
                         : launch(mid_seg_kernel<Op, false, false, 4>, none);
    if (ctas == 6)
        return inclusive ? launch(mid_seg_kernel<Op, true, false, k6>, none)
                         : launch(mid_seg_kernel<Op, false, false, k6>, none);
    return inclusive ? launch(mid_seg_kernel<Op, true, false, kMost>, none)
                     : launch(mid_seg_kernel<Op, false, false, kMost>, none);
}

}  // namespace gps
