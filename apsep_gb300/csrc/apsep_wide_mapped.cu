// apsep_wide_mapped.cu -- the consumers' forms of the range engine for 8-byte
// keys: the order-reversing key map (previous greater, and the stock span with
// the span output form) and the reversed array (next smaller), as for 4-byte keys
// (apsep_mapped.cu), in the 512-key tiles of long arrays (16 keys per lane, 12
// warps per CTA; wide_tile_keys).  Shorter arrays take a flip or reverse pass and
// a plain run: a pass over so few keys costs little more than its launch.
// Single arrays on a 16-byte boundary (keys and answers).  A pass over 8-byte keys
// less (2^24 + 5 uniform int64 keys, us, pass and plain run | this run): previous
// greater 131 | 96, stock span 151 | 100, next smaller 156 | 115, Cartesian parents
// 279 | 244; float64 144 | 108, 173 | 113, 167 | 126, 314 | 271.
#include "apsep_range_kernel.cuh"

namespace apsep {

namespace {
constexpr int kIpt = 16, kWpc = 12;
constexpr int kMaxDevWM = 64;
int g_warps_wm[kMaxDevWM];  // resident warps per device

// The kernels of one key type: FWD its key map, FLIP the order-reversing one.
template <int FWD, int FLIP>
struct Forms {
    static cudaError_t prepare(int* per_sm) {
        cudaError_t rr[5] = {prepare_t<int64_t, kIpt, kWpc, false, false, true, FLIP, OUT_I32>(per_sm),
                             prepare_t<int64_t, kIpt, kWpc, true, false, true, FLIP, OUT_I32>(per_sm),
                             prepare_t<int64_t, kIpt, kWpc, false, false, true, FLIP, OUT_SPAN>(per_sm),
                             prepare_t<int64_t, kIpt, kWpc, false, false, true, FWD, OUT_I32, true>(per_sm),
                             prepare_t<int64_t, kIpt, kWpc, true, false, true, FWD, OUT_I32, true>(per_sm)};
        for (int q = 0; q < 5; q++)
            if (rr[q] != cudaSuccess) return rr[q];
        return cudaSuccess;
    }
    static cudaError_t flipped(int incl, int span, RangeArgs& a, const CUtensorMap& mi, const CUtensorMap& mo,
                               cudaStream_t st, int mw) {
        if (span) return launch_t<int64_t, kIpt, kWpc, false, false, true, FLIP, OUT_SPAN>(a, mi, mo, st, mw);
        return incl ? launch_t<int64_t, kIpt, kWpc, true, false, true, FLIP, OUT_I32>(a, mi, mo, st, mw)
                    : launch_t<int64_t, kIpt, kWpc, false, false, true, FLIP, OUT_I32>(a, mi, mo, st, mw);
    }
    static cudaError_t reversed(int incl, RangeArgs& a, const CUtensorMap& mi, const CUtensorMap& mo, cudaStream_t st,
                                int mw) {
        return incl ? launch_t<int64_t, kIpt, kWpc, true, false, true, FWD, OUT_I32, true>(a, mi, mo, st, mw)
                    : launch_t<int64_t, kIpt, kWpc, false, false, true, FWD, OUT_I32, true>(a, mi, mo, st, mw);
    }
};
using Int = Forms<KMAP_NONE, KMAP_FLIP>;
using Float = Forms<KMAP_F64, KMAP_F64_FLIP>;

cudaError_t warps_for(int* warps) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevWM) return cudaErrorInvalidValue;
    if (!g_warps_wm[dev]) {
        int per_sm = 0, sms = 0;
        if ((e = Int::prepare(&per_sm)) != cudaSuccess) return e;
        if ((e = Float::prepare(&per_sm)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorInvalidConfiguration;
        const int w = per_sm * sms * kWpc;
        g_warps_wm[dev] = w > kMaxRanges ? kMaxRanges : w;
    }
    *warps = g_warps_wm[dev];
    return cudaSuccess;
}
}  // namespace

cudaError_t launch_wide_flipped(int dtype, int incl, int span, RangeArgs& a, const CUtensorMap& mi,
                                const CUtensorMap& mo, cudaStream_t st) {
    int mw = 0;
    const cudaError_t e = warps_for(&mw);
    if (e != cudaSuccess) return e;
    if (a.head != 0 || dtype < 2 || (span && incl)) return cudaErrorInvalidValue;
    return dtype == 2 ? Int::flipped(incl, span, a, mi, mo, st, mw) : Float::flipped(incl, span, a, mi, mo, st, mw);
}

cudaError_t launch_wide_reversed(int dtype, int incl, RangeArgs& a, const CUtensorMap& mi, const CUtensorMap& mo,
                                 cudaStream_t st) {
    int mw = 0;
    const cudaError_t e = warps_for(&mw);
    if (e != cudaSuccess) return e;
    if (a.head != 0 || dtype < 2 || (a.tma_rows > 0 && (int64_t)a.tma_rows * 16 != (int64_t)a.n))
        return cudaErrorInvalidValue;
    return dtype == 2 ? Int::reversed(incl, a, mi, mo, st, mw) : Float::reversed(incl, a, mi, mo, st, mw);
}

}  // namespace apsep
