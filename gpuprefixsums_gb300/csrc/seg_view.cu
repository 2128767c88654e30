// Generic scan of u32 and u64 buffers off a 16-byte boundary (scan_seg.cuh, VIEW).
#include "seg_launch.cuh"

namespace gps {
namespace {

template <class Op>
cudaError_t launch_view_t(bool inclusive, const ScanArgs& a0, int num_sms, cudaStream_t stream, LaunchInfo* info) {
    using T = typename Op::T;
    constexpr uint32_t EPC = 16 / sizeof(T), TILE = 16384 / sizeof(T);
    auto phase = [](const void* p) { return static_cast<uint32_t>((reinterpret_cast<uintptr_t>(p) & 15u) / sizeof(T)); };
    ScanArgs a = a0;
    a.view_lead = phase(a0.in);
    a.view_shift = (phase(a0.out) + EPC - a.view_lead) % EPC;
    a.in = static_cast<const T*>(a0.in) - a.view_lead;
    a.out = static_cast<T*>(a0.out) - (a.view_lead + a.view_shift);
    a.n = a0.n + a.view_lead;
    // At most one tile more than on aligned buffers: a quarter of a unit.
    a.num_tiles = static_cast<uint32_t>((a.n + a.view_shift + TILE - 1) / TILE);
    const SegArgs none{nullptr, 0};
    const GenericConfig cfg = kGenericCandidates[0];
    return inclusive ? launch_seg_t<Op, true, false, 4, 1, true>(a, none, cfg, num_sms, stream, info)
                     : launch_seg_t<Op, false, false, 4, 1, true>(a, none, cfg, num_sms, stream, info);
}

}  // namespace

cudaError_t launch_seg_view(gps_dtype dtype, bool inclusive, const ScanArgs& a, int num_sms, cudaStream_t stream,
                            LaunchInfo* info) {
    return dtype == GPS_DTYPE_U64 ? launch_view_t<OpU64>(inclusive, a, num_sms, stream, info)
                                  : launch_view_t<OpU32>(inclusive, a, num_sms, stream, info);
}

}  // namespace gps
