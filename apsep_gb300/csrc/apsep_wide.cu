// apsep_wide.cu -- the range engine for 8-byte keys (int64 / float64).
//
// The same kernel template with 8-byte keys, keys streamed as 128-byte TMA rows
// of 16 keys, answers as int32 positions (n < 2^31).
// No 64-bit key fits beside a tag in one atomic word, so the tagged words hold
// the tag alone and group minima are read from the ranges' minima.
// float64 keys run as int64 through an order-preserving map of their bits
// (applied as keys are read into registers): the FP64 compare rate
// of this part would make every comparison the bottleneck.
// Single arrays and segmented batches; two shapes, chosen by the length
// (wide_tile_keys); no view head (arrays off a 16-byte boundary take plain
// loads and stores).
#include "apsep_range_kernel.cuh"

namespace apsep {

namespace {
// Shape 0: 8 keys per lane, 8 warps per CTA, two CTAs per SM.  Shape 1: 16 keys
// per lane, 12 warps per CTA, one CTA per SM.  What a tile costs whatever its
// length (the lane ladder's top, the cross-lane queries, the ring's waits) is most
// of the instructions, and twice the keys per tile pay it half as often.  Shape 1's
// warps take 18 KB each, so an SM holds 12 of them against 16.
constexpr int kIpt0 = 8, kWpc0 = 8;
constexpr int kIpt1 = 16, kWpc1 = 12;
constexpr int kMaxDevW = 64;
int g_wide_warps[kMaxDevW][2];  // resident warps per device and shape
int g_wide_sms[kMaxDevW];

template <int IPT, int WPC, bool SEG>
cudaError_t prep(int* per_sm) {
    cudaError_t rr[4] = {prepare_t<int64_t, IPT, WPC, false, SEG, !SEG>(per_sm),
                         prepare_t<int64_t, IPT, WPC, true, SEG, !SEG>(per_sm),
                         prepare_t<int64_t, IPT, WPC, false, SEG, !SEG, KMAP_F64>(per_sm),
                         prepare_t<int64_t, IPT, WPC, true, SEG, !SEG, KMAP_F64>(per_sm)};
    for (int q = 0; q < 4; q++)
        if (rr[q] != cudaSuccess) return rr[q];
    return cudaSuccess;
}

template <int IPT, int WPC, bool SEG>
cudaError_t launch_wide(int dtype, int incl, RangeArgs& a, const CUtensorMap& mi, const CUtensorMap& mo,
                        cudaStream_t st, int max_warps) {
    if (dtype == 2)
        return incl ? launch_t<int64_t, IPT, WPC, true, SEG, !SEG>(a, mi, mo, st, max_warps)
                    : launch_t<int64_t, IPT, WPC, false, SEG, !SEG>(a, mi, mo, st, max_warps);
    // float64: int64 slots compared through the order map (no FP64 compares)
    return incl ? launch_t<int64_t, IPT, WPC, true, SEG, !SEG, KMAP_F64>(a, mi, mo, st, max_warps)
                : launch_t<int64_t, IPT, WPC, false, SEG, !SEG, KMAP_F64>(a, mi, mo, st, max_warps);
}
}  // namespace

cudaError_t prepare_wide() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevW) return cudaErrorInvalidValue;
    if (g_wide_sms[dev]) return cudaSuccess;
    int per_sm[2] = {0, 0};
    if ((e = prep<kIpt0, kWpc0, false>(&per_sm[0])) != cudaSuccess) return e;
    if ((e = prep<kIpt0, kWpc0, true>(&per_sm[0])) != cudaSuccess) return e;
    if ((e = prep<kIpt1, kWpc1, false>(&per_sm[1])) != cudaSuccess) return e;
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (per_sm[0] < 1 || per_sm[1] < 1) return cudaErrorInvalidConfiguration;
    const int w0 = per_sm[0] * sms * kWpc0, w1 = per_sm[1] * sms * kWpc1;
    g_wide_warps[dev][0] = w0 > kMaxRanges ? kMaxRanges : w0;
    g_wide_warps[dev][1] = w1 > kMaxRanges ? kMaxRanges : w1;
    g_wide_sms[dev] = sms;
    return cudaSuccess;
}

// Keys per warp tile of one run on the current device (0: no device).  Single
// arrays take shape 1 once shape 0 would need a second CTA on some SM (n > 311,296
// here).  Up to there every warp has one tile in either shape, and the shorter tile
// is the shorter chain; past it shape 0's warps share their SM's issue slots.  int64
// keys, shape 0 against shape 1, us: 2^17 uniform 12.4 | 13.4, nearly sorted
// descending 17.3 | 19.8; 300,001 keys 14.2 | 15.7 and 26.5 | 26.5; 330,001 keys
// 15.3 | 15.0 and 31.1 | 24.9; 2^19 18.7 | 15.1 and 40.3 | 29.7; 2^22 43.6 | 35.3
// and 56.2 | 49.0; 2^25 218 | 168 and 128 | 119; random walks, whose long lists of
// phase 2 have fewer warps to share, 2^20 35 | 42, 2^22 76 | 70, 2^25 365 | 329.
// Arrays off a 16-byte boundary, which take plain loads, keep shape 0 and its 16 warps
// (2^24 int64 keys, shape 0 against shape 1, us: uniform 201 | 226, descending
// 139 | 169, ascending 144 | 175).
// Batches keep shape 0 (2^25 keys in 1024 segments: uniform 237 | 184, but a walk
// 404 | 486), as do the pieces of the int64-position path (2^27 keys in two: uniform
// 970 | 800, walk 1816 | 1906; 2^24 in two: descending 163 | 197).
int wide_tile_keys(int64_t n, bool segmented, bool aligned) {
    int dev = 0;
    if (prepare_wide() != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (segmented || !aligned) return 32 * kIpt0;
    return n > (int64_t)32 * kIpt0 * kWpc0 * g_wide_sms[dev] ? 32 * kIpt1 : 32 * kIpt0;
}

cudaError_t launch_range_wide(int dtype, int incl, int tile_keys, RangeArgs& a, const CUtensorMap& mi,
                              const CUtensorMap& mo, cudaStream_t st) {
    cudaError_t e = prepare_wide();
    if (e != cudaSuccess) return e;
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    a.head = 0;
    if (a.offsets) {  // a segmented batch
        if (a.nseg < 1 || tile_keys != 32 * kIpt0) return cudaErrorInvalidValue;
        return launch_wide<kIpt0, kWpc0, true>(dtype, incl, a, mi, mo, st, g_wide_warps[dev][0]);
    }
    a.nseg = 0;
    if (tile_keys == 32 * kIpt1)
        return launch_wide<kIpt1, kWpc1, false>(dtype, incl, a, mi, mo, st, g_wide_warps[dev][1]);
    if (tile_keys != 32 * kIpt0) return cudaErrorInvalidValue;
    return launch_wide<kIpt0, kWpc0, false>(dtype, incl, a, mi, mo, st, g_wide_warps[dev][0]);
}

}  // namespace apsep
