// Internal definitions shared by the scan kernels and the C ABI layer:
// the device workspace header, the tile-descriptor encodings and the kernel
// argument block.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "gps.h"

namespace gps {

// Tile ids handed out by the producer; kTileEnd marks "no more tiles".
constexpr uint32_t kTileEnd = 0xFFFFFFFFu;

// Epochs are 30 bits wide so that they fit beside a 32-bit value in a 64-bit
// descriptor. Epoch 0 never occurs, so a zeroed workspace is "not ready".
constexpr uint32_t kEpochMask = 0x3FFFFFFFu;

// Descriptor slots allocated past the last tile: a lookback window is read in
// aligned groups of up to 16 slots and may end up to 15 slots after its tile.
constexpr uint32_t kDescPad = 16;

// Descriptor status (two bits), as in the decoupled-lookback scheme:
// not ready / tile aggregate only / inclusive prefix through this tile.
enum DescStatus : uint32_t { kNotReady = 0, kAggregate = 1, kInclusive = 2 };

// Bits of WsHeader::error_flags.
enum ErrFlag : uint32_t {
    kErrLookbackTimeout = 1u,  // a lookback spin ran past its wait budget
    kErrPipelineTimeout = 2u,  // an mbarrier wait ran past its wait budget
    kErrStallTimeout = 4u,     // a forced-stall wait ran past its wait budget
};

// Device-resident state of one plan. Zeroed at plan creation, then epoch=1.
// tile_counter / exit_counter are returned to zero by the last CTA of every
// launch, and the same CTA advances the epoch, so consecutive launches need no
// memset and a launch can be replayed from a CUDA graph.
struct alignas(128) WsHeader {
    uint32_t tile_counter;
    uint32_t exit_counter;
    uint32_t epoch;
    uint32_t error_flags;
    // One-tile-per-CTA kernels: their launch number and how many of the launches
    // used the group sums, read by one 16-byte load. A CTA publishes only what rests
    // on that load, so none can still be about to read either word once the last
    // tile, which has seen every other, advances them.
    alignas(16) uint64_t mid_launch;
    uint32_t sums_launch;  // mod 2^32: only its lowest bit counts
    uint32_t pad_;
    unsigned long long capacity_tiles;  // descriptor slots that follow
    unsigned long long stat_polls;      // lookback windows re-polled (stats mode)
    unsigned long long stat_fallbacks;  // predecessor tiles re-reduced
    unsigned long long stat_inserts;    // fallback aggregates that won the CAS
    unsigned long long stat_stalls;     // tiles that were made to stall
};
static_assert(sizeof(WsHeader) == 128, "header is one 128-byte line");
static_assert(offsetof(WsHeader, mid_launch) % 16 == 0 &&
                  offsetof(WsHeader, sums_launch) == offsetof(WsHeader, mid_launch) + 8,
              "launch number and set count are one 16-byte word");

// Forced-stall test mode (EmulatedDeadlocking-style).
//  mode 0: off.
//  mode 1: every tile with (t % period) == 0 stalls (the reference pattern).
//  mode 2: tiles selected by a seeded hash with probability 1/period stall.
// A stalled tile withholds its aggregate for up to delay_ns or until a
// successor re-reduces its input and inserts the aggregate for it
// (fallback_polls > 0 enables that fallback after this many empty polls).
struct StallConfig {
    uint32_t mode;
    uint32_t period;
    uint32_t seed;
    uint32_t delay_ns;
    uint32_t fallback_polls;
    uint32_t pad_;
};

// Fixed-order lookback of the generic kernel (scan_seg.cuh): lookback units
// per group, and the group descriptors a plan keeps for up to `units` units
// (one more than the groups, as slack).
constexpr uint32_t det_group_units(int unit_tiles, bool long_groups) {
    return unit_tiles == 1 || long_groups ? 128u : 64u;
}
constexpr uint64_t det_group_slots(uint64_t units) { return (units + 63) / 64 + 1; }

// The generic kernel's unit and group descriptors sit one per 128-byte line
// (a stride of 8 words) when a launch has at most kSegStrideMaxUnits
// lookback units, else packed (Op::kDescWords words each). Measured on GB300
// (FP32, GPU time per scan): one per line 11.6 against 12.4 us at 2^20, 14.9
// against 15.7 at 2^22, 29.0 against 31.7 at 2^24 (1024 units of 4 tiles);
// packed 91 against 94 us at 2^26 and 173 against 178 at 2^27, where the
// wider reads compete with the data for L2. 16-byte words a plan keeps for
// up to `tiles` units of `dw` words, and for their group descriptors:
constexpr uint32_t kSegDescStride = 8;
constexpr uint64_t kSegStrideMaxUnits = 1024;
constexpr uint64_t seg_desc_words(uint64_t tiles, uint64_t dw) {
    const uint64_t packed = (tiles + kDescPad) * dw;
    const uint64_t strided = ((tiles < kSegStrideMaxUnits ? tiles : kSegStrideMaxUnits) + kDescPad) * kSegDescStride;
    return packed > strided ? packed : strided;
}
constexpr uint64_t seg_group_words(uint64_t tiles, uint64_t dw) {
    const uint64_t packed = det_group_slots(tiles) * dw;
    const uint64_t strided = det_group_slots(tiles < kSegStrideMaxUnits ? tiles : kSegStrideMaxUnits) * kSegDescStride;
    return packed > strided ? packed : strided;
}

struct ScanArgs {
    const void* in;
    void* out;
    uint64_t n;
    uint32_t num_tiles;
    // One-tile-per-CTA and generic kernels: 16-byte words from one descriptor
    // to the next (0: packed), set by their launchers.
    uint32_t desc_stride;
    // Plan state (counters, epoch, error flags). Kernels that share descriptors share a
    // header, the one-tile-per-CTA kernels the one with their launch number: after a wait
    // that ran out the number may stay, and what one of them has published under it is not
    // to be taken for another's.
    WsHeader* hdr;
    void* desc;          // tile descriptors (lookback)
    // Descriptors of groups: of kMidSegGroup tiles for the one-tile-per-CTA form
    // of the generic kernel, of det_group_units() lookback units for the other. For
    // mid.cu: two sets of kMidSums 128-byte lines, and two 16-byte carries.
    void* group_desc;
    const void* carry_in;  // optional: one element added to every output
    void* carry_out;       // optional: receives carry_in + sum of all n inputs
    uint64_t wait_budget_ns;
    StallConfig stall;
    uint64_t* mid_launch;  // one-tile-per-CTA kernels: WsHeader::mid_launch, sums_launch after it
    uint32_t units_in_flight;  // generic kernel: per CTA, set by its launcher
    // Generic kernel on buffers off a 16-byte boundary (its launcher sets them):
    // elements before the input in its first 16 bytes, and how many elements
    // further the outputs sit from their boundary.
    uint32_t view_lead, view_shift;
};

// Kernel geometry shared by host and device: RW reduce warps and RW finalize
// warps, each thread of either owning 128 contiguous bytes of the tile, plus
// one producer warp and kLookbackWarps lookback warps per CTA.
template <typename T, int RW>
struct TileShape {
    static constexpr int kItems = 128 / static_cast<int>(sizeof(T));
    static constexpr int kRoleThreads = RW * 32;
    static constexpr int kTile = kRoleThreads * kItems;
    static constexpr int kLookbackWarps = 2;
    static constexpr int kThreads = 32 * (1 + kLookbackWarps + 2 * RW);
};

// Segments of a batched (segmented) scan: segment s is
// [offsets[s], offsets[s+1]); offsets has num_segments + 1 entries.
struct SegArgs {
    const uint32_t* offsets;
    uint32_t num_segments;
};

// ------------------------------------------------------------ launchers
// Each returns the launch status; they never synchronize.
struct LaunchInfo {
    int grid;
    int block;
    size_t smem;
    uint32_t launches = 1;
};

cudaError_t launch_csdl(gps_dtype dtype, bool inclusive, bool stall_mode, const ScanArgs& a,
                        int num_sms, cudaStream_t stream, LaunchInfo* info);
// Sets up, without launching, every kernel launch_csdl() can pick for this
// dtype without forced stalls, so that later launches make no set-up call.
cudaError_t prepare_csdl(gps_dtype dtype);
cudaError_t launch_rts(gps_dtype dtype, bool inclusive, const ScanArgs& a, void* scratch,
                       int num_sms, cudaStream_t stream, LaunchInfo* info);
// Elements of scratch a reduce-then-scan plan keeps, and the kernel launches
// of a scan of n elements of an aligned buffer.
uint64_t rts_scratch_elems(int num_sms);
uint32_t rts_launches(uint64_t n, uint32_t tile_elems, int num_sms);
// Tensor maps of the generic kernel: the buffer seen as rows of 128 bytes
// (32 four-byte or 16 eight-byte elements), boxes of 128 rows (one 16 KB
// tile), 128-byte swizzle. Rows past the last full row are the kernel's to
// handle with plain loads and stores. Host-side; encodes through the driver
// entry point cuTensorMapEncodeTiled.
struct RowMaps {
    CUtensorMap in;
    CUtensorMap out;
};
// (of n elements of input and out_n of output).
cudaError_t encode_row_maps(const void* in, void* out, uint64_t n, uint64_t out_n, uint32_t elem_size, RowMaps* maps);

// Launch configuration of the generic kernel: tiles per lookback unit (1 or
// 4; the unit is what one CTA takes from the work counter), the CTA count as
// a fraction of the resident maximum (1 = all, 2 = half), and threads per
// 128-byte row of a tile (1: 4 reduce warps and two groups of 4 finalize warps,
// each thread scanning 128 bytes; 2: 8 and 8, each thread scanning 64 bytes). A unit of 0
// stands for one tile per CTA (mid_seg.cuh).
struct GenericConfig {
    uint32_t unit;
    uint32_t ctas_div;
    uint32_t split;
};
// The first is the untuned choice above the sizes of one tile per CTA: every SM has a
// unit of 4 tiles there. Measured on GB300, units of 4 tiles against single-tile units, batched
// u32: 640 tiles 11.7 / 13.1 us, 1024 tiles 13.5 / 16.3.
constexpr GenericConfig kGenericCandidates[] = {{4, 1, 1}, {1, 1, 1}, {4, 2, 1}, {1, 2, 1},
                                                {4, 1, 2}, {1, 1, 2}, {4, 2, 2}, {1, 2, 2}};
constexpr int kNumGenericCandidates = 8;
// Whether a plain u32 or u64 scan above the mid size runs on the generic kernel.
bool integer_scan_takes_generic(uint64_t n, uint32_t tiles, int num_sms);

// Generic single-pass scan (scan_seg.cuh), one per scan operation; `sg` null
// for a plain scan. Buffers must be 16-byte aligned; descriptors are 16 bytes.
cudaError_t launch_seg_u32(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg, int num_sms,
                           cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_u64(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg, int num_sms,
                           cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_f32(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg, int num_sms,
                           cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_f32c(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                            int num_sms, cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_u32x4(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                             int num_sms, cudaStream_t stream, LaunchInfo* info);
// Plain u32 and u64 scans of buffers off a 16-byte boundary, in units of 4 tiles
// (seg_view.cu).
cudaError_t launch_seg_view(gps_dtype dtype, bool inclusive, const ScanArgs& a, int num_sms, cudaStream_t stream,
                            LaunchInfo* info);
// The same with two threads per row (cfg.split == 2), in translation units of
// their own (seg_*_x2.cu); cudaErrorNotSupported when that kernel shape does
// not fit one CTA's shared memory for the type.
cudaError_t launch_seg_u32_x2(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                              int num_sms, cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_u64_x2(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                              int num_sms, cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_f32_x2(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                              int num_sms, cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_f32c_x2(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                               int num_sms, cudaStream_t stream, LaunchInfo* info);
cudaError_t launch_seg_u32x4_x2(bool inclusive, const ScanArgs& a, const SegArgs* sg, const GenericConfig& cfg,
                                int num_sms, cudaStream_t stream, LaunchInfo* info);
// Whether the two-threads-per-row kernels of a unit size fit one CTA.
bool seg_u32_x2_fits(uint32_t unit);
bool seg_u64_x2_fits(uint32_t unit);
bool seg_f32_x2_fits(uint32_t unit);
bool seg_f32c_x2_fits(uint32_t unit);
bool seg_u32x4_x2_fits(uint32_t unit);

// Stream compaction by flag bytes (select.cu): elements per tile for an
// element size, and the launch. a.carry_out receives the count (uint64).
uint32_t select_tile_elems(size_t elem_size);
// Selects of up to this many tiles run one tile per CTA, on the plan's
// mid-size descriptors: where that met the persistent kernel before its lookback came
// down to one round trip. Measured since (152 SMs, graph replay, inputs from HBM, us, against the
// persistent kernel): u32, 30% selected, 2400 tiles 15.6 / 20.3, 2500 17.5 / 20.6, 3200
// 20.2 / 23.8, 4095 25.7 / 25.7; u64 2500 17.7 / 19.2, 3200 20.2 / 22.0; 10% and 90% alike. The two
// meet at about 4095 tiles now; the limit stands where it was.
constexpr uint32_t kMidSelectMaxTiles = 2500;
cudaError_t launch_select(size_t elem_size, const ScanArgs& a, const uint8_t* flags, int num_sms, cudaStream_t stream,
                          LaunchInfo* info);

// Small integer scans in one CTA (small.cu): up to kSmallMaxBytes of input.
constexpr size_t kSmallMaxBytes = 64 * 1024;
uint64_t small_scan_max_elems(gps_dtype dtype);
cudaError_t launch_small(gps_dtype dtype, bool inclusive, const ScanArgs& a, cudaStream_t stream, LaunchInfo* info);

// Integer chained scans up to mid size, one 16 KB tile per CTA (mid.cu); the
// default upper size of a plan: 2448 tiles, one limit for three curves. Measured on GB300
// (152 SMs: two waves of 8 CTAs per SM are 2432 tiles; graph replay, inputs from HBM, us)
// against the generic kernel, which takes over: u32 2400 tiles 17.4 / 18.9, 2440 18.0 / 18.7, 2448
// 19.0 / 18.8, 2500 19.9 / 18.8; off a 16-byte boundary 2400 20.0 / 20.2, 2432 20.4 / 20.3, 2448
// 21.3 / 20.5; u64 2300 18.3 / 18.1, 2400 19.1 / 18.6, 2448 19.9 / 18.6: u32 meets it at the limit, views
// 30 tiles below, u64 some 150 below. Earlier measurements had all three within 30 tiles of it.
constexpr size_t mid_max_bytes() { return 153ull << 18; }
// Tile descriptors of the one-tile-per-CTA kernels sit one per 128-byte line
// (a stride of 8 words) when a launch has more than one group of 32 tiles, else
// packed. Sharing lines between
// tiles that publish and read at the same moment cost up to 3 us per read
// (2^20 u32: 6.04 us packed, 4.95 us one per line, 5.23 us one per 32-byte
// sector); with one group, packed reads are faster (2^17: 2.83 against
// 3.36 us). Group sums and group descriptors always take a line each. A launch
// takes at most kMidMaxTiles tiles. Tile-descriptor words a plan keeps for
// `tiles` tiles:
constexpr uint32_t kMidDescStride = 8;
constexpr uint64_t kMidMaxTiles = 4096;
constexpr uint64_t mid_desc_words(uint64_t tiles) {
    return ((tiles < kMidMaxTiles ? tiles : kMidMaxTiles) + kDescPad) * kMidDescStride;
}
// Group sums of the integer kernel: two sets, 128 bytes a group.
constexpr uint32_t kMidSums = 128;
// One-tile-per-CTA form of the generic kernel (mid_seg.cuh): tiles per group
// of its lookback, and the most tiles it takes.
constexpr uint32_t kMidSegGroup = 64;
constexpr uint32_t kMidSegMaxTiles = 4096;
static_assert(kMidSegGroup >= 32 && kMidSegMaxTiles <= kMidMaxTiles, "within the plan's mid-size descriptors");
constexpr GenericConfig kMidSegConfig = {0, 1, 1};
// Untuned scans of up to this many tiles take it; larger ones the kernel with
// units, whose pipeline then pays. The wider the running state, the fewer CTAs
// an SM holds and the longer each takes. Measured on GB300 (152 SMs, for which these are
// constants; graph replay, inputs from HBM, us, one tile per CTA against units of 4 tiles): FP32
// 1728 tiles 14.8 / 15.9, 1900 15.8 / 16.4, 2048 16.9 / 16.6; batched u32 1900 tiles 16.3 / 17.6,
// 2048 17.3 / 17.9, 2200 18.1 / 18.6; compensated 1250 tiles 13.8 / 14.6, 1400 16.0 / 16.0, batched
// 1728 tiles 18.7 / 20.2, 2048 21.7 / 22.0; batched u64 1728 tiles 15.9 / 16.9, 1900 17.4 / 17.5, 2048
// 18.6 / 17.7; structs 640 tiles 10.8 / 11.8, 720 11.4 / 11.0, batched 11.6 / 12.0 and 11.7 / 11.8.
constexpr uint64_t mid_seg_default_tiles(gps_dtype dtype, bool segmented) {
    switch (dtype) {
        case GPS_DTYPE_U32:
        case GPS_DTYPE_F32: return 2048;
        case GPS_DTYPE_U64: return 1728;
        case GPS_DTYPE_F32_COMPENSATED: return segmented ? 1728 : 1280;
        case GPS_DTYPE_U32X4: break;
    }
    return 704;
}
// Launches of a scan of n elements of an aligned buffer by the integer kernel.
constexpr uint32_t mid_launches(uint64_t n, uint32_t tile_elems) {
    return static_cast<uint32_t>((n + kMidMaxTiles * tile_elems - 1) / (kMidMaxTiles * tile_elems));
}
cudaError_t launch_mid(gps_dtype dtype, bool inclusive, const ScanArgs& a, int num_sms, cudaStream_t stream,
                       LaunchInfo* info);

uint32_t csdl_tile_elems(gps_dtype dtype);
// Sets the text gps_last_error() returns on this host thread.
void record_error(const char* msg);
uint32_t rts_tile_elems(gps_dtype dtype);
size_t dtype_size(gps_dtype dtype);

}  // namespace gps
