// A 16 KB tile as four rows of 256 16-byte chunks, for CTAs of 256 threads:
// thread tid holds chunk tid of every row, so each warp load or store moves
// 512 contiguous bytes.
//
// ALIGNED = false takes buffers at any element offset from a 16-byte
// boundary. Tiles are then counted from the boundary at or below the input
// ("virtual" index j = i + lead, lead elements of tile 0 lying before the
// input), so every load but those of the first and last chunk stays a 16-byte
// one. The output's boundary may lie elsewhere: if virtual element 0 sits
// `phase` elements past one, an output chunk is the last `phase` elements of
// the chunk on the left (one shuffle each) and the first of this one, stored
// as 16 bytes; a warp's two edges, tile 0 and a partial tile store elements.
#pragma once
#include "scan_pipeline.cuh"

namespace gps {

constexpr int kRowThreads = 256;

// How chunks are read and written: through L1, or past it with an L2 policy.
struct PlainAccess {
    template <typename T>
    __device__ __forceinline__ Chunk<T> ld(const T* p) const {
        return *reinterpret_cast<const Chunk<T>*>(p);
    }
    template <typename T>
    __device__ __forceinline__ void st(T* p, const Chunk<T>& q) const {
        *reinterpret_cast<Chunk<T>*>(p) = q;
    }
};
struct PolicyAccess {
    uint64_t policy;
    template <typename T>
    __device__ __forceinline__ Chunk<T> ld(const T* p) const {
        const uint4 v = ptx::ld_policy_v4(p, policy);
        return *reinterpret_cast<const Chunk<T>*>(&v);
    }
    template <typename T>
    __device__ __forceinline__ void st(T* p, const Chunk<T>& q) const {
        ptx::st_policy_v4(p, *reinterpret_cast<const uint4*>(&q), policy);
    }
};

template <typename T, bool ALIGNED>
struct TileRows {
    static constexpr int kTile = 16384 / static_cast<int>(sizeof(T));
    static constexpr int kEpc = 16 / static_cast<int>(sizeof(T));
    static constexpr int kRow = kRowThreads * kEpc;
    static constexpr int kRows = kTile / kRow;  // 4

    const T* src;  // this thread's chunk of row 0
    T* dst;
    uint32_t off0;   // its first element within the tile
    uint32_t first;  // elements of the tile before it do not exist
    uint32_t cnt;    // nor from here on
    bool full;

    __host__ __device__ static uint32_t lead_of(const void* in) {
        return ALIGNED ? 0u : static_cast<uint32_t>((reinterpret_cast<uintptr_t>(in) & 15u) / sizeof(T));
    }
    // Tiles of a scan of n elements: at most one more than on aligned buffers.
    static uint32_t tiles(const void* in, uint64_t n) {
        return static_cast<uint32_t>((n + lead_of(in) + kTile - 1) / kTile);
    }

    __device__ TileRows(const void* in, void* out, uint64_t n, uint32_t t, uint32_t tid) {
        const uint64_t t0 = static_cast<uint64_t>(t) * kTile;
        const uint32_t lead = lead_of(in);
        off0 = tid * kEpc;
        first = t == 0 ? lead : 0u;
        cnt = static_cast<uint32_t>(min(static_cast<uint64_t>(kTile), n + lead - t0));
        full = cnt == static_cast<uint32_t>(kTile) && first == 0;
        src = static_cast<const T*>(in) - lead + t0 + off0;
        dst = static_cast<T*>(out) - lead + t0 + off0;
    }

    __device__ __forceinline__ bool whole(uint32_t off) const {
        return full || (off >= first && off + kEpc <= cnt);
    }

    template <class Access>
    __device__ __forceinline__ Chunk<T> load(int r, Access access) const {
        const uint32_t off = r * kRow + off0;
        Chunk<T> q;
        if (whole(off)) {
            q = access.ld(src + r * kRow);
        } else {
#pragma unroll
            for (int e = 0; e < kEpc; ++e) q.v[e] = off + e >= first && off + e < cnt ? src[r * kRow + e] : T(0);
        }
        return q;
    }

    // A warp's row of chunks whose output lies P elements past a boundary.
    template <int P, class Access>
    __device__ __forceinline__ static void put_shifted(T* p, uint32_t lane, const Chunk<T>& q, Access access) {
        Chunk<T> w;
#pragma unroll
        for (int e = 0; e < kEpc; ++e) {
            if (e < P)
                w.v[e] = __shfl_up_sync(kFullMask, q.v[kEpc - P + e], 1);
            else
                w.v[e] = q.v[e - P];
        }
        if (lane != 0) {
            access.st(p - P, w);
        } else {
#pragma unroll
            for (int e = 0; e < kEpc - P; ++e) p[e] = q.v[e];
        }
        if (lane == 31) {
#pragma unroll
            for (int e = kEpc - P; e < kEpc; ++e) p[e] = q.v[e];
        }
    }

    // By whole warps.
    template <class Access>
    __device__ __forceinline__ void store(int r, const Chunk<T>& q, uint32_t lane, Access access) const {
        const uint32_t off = r * kRow + off0;
        T* p = dst + r * kRow;
        const uint32_t phase =
            ALIGNED ? 0u : static_cast<uint32_t>((reinterpret_cast<uintptr_t>(p) & 15u) / sizeof(T));
        if (phase == 0 && whole(off)) {
            access.st(p, q);
        } else if (phase == 0 || !full) {
#pragma unroll
            for (int e = 0; e < kEpc; ++e)
                if (off + e >= first && off + e < cnt) p[e] = q.v[e];
        } else if (phase == 1) {
            put_shifted<1>(p, lane, q, access);
        } else if (kEpc == 4 && phase == 2) {
            put_shifted<kEpc == 4 ? 2 : 1>(p, lane, q, access);
        } else {
            put_shifted<kEpc == 4 ? 3 : 1>(p, lane, q, access);
        }
    }
};

}  // namespace gps
