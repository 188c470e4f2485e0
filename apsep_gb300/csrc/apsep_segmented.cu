// apsep_segmented.cu -- the segmented instantiations of the range engine.
//
// A batch of arrays stored back to back (segment s is d_in[off[s],
// off[s+1])) runs as one launch over the concatenation: every key's answer is
// the nearest earlier key that qualifies in the whole concatenation, turned
// relative to its own segment start -- and -1 when that key lies before the
// segment, since then nothing in the segment qualifies.  The kernel follows
// the segment starts tile by tile (apsep_range_kernel.cuh, step 0), converts
// the tile's answers before its store, and skips the cross-range search for
// any deferred key whose segment starts inside its own range.
#include "apsep_range_kernel.cuh"

namespace apsep {

cudaError_t prepare_segmented(int cfg, int* ctas_per_sm) { return prepare_mode<true, false>(cfg, ctas_per_sm); }

cudaError_t launch_range_segmented(int dtype, int incl, int cfg, RangeArgs& a, const CUtensorMap& mi,
                                   const CUtensorMap& mo, cudaStream_t st) {
    int max_warps = 0;
    cudaError_t e = range_max_warps(cfg, &max_warps);
    if (e != cudaSuccess) return e;
    if (cfg == 0) {
        // One CTA of 20 warps per SM instead of 16: a batch has no whole-tile paths for
        // sorted keys, which lose to the finer ranges (2^25 descending 54 -> 58 us as a
        // single array), and hides more of its dependent steps: 1.03e8 keys in 1024
        // arrays, mixed 410 -> 379 us, uniform 316 -> 305, sawtooth 338 -> 305.  Below
        // six tiles a range the finer ranges cost more than they hide (8.2e6 keys 69.6
        // us; 1.35e7 keys 95.0): those take configuration 2, 16 warps per SM in two CTAs
        // (67.0; 97.7).
        int dev = 0, sms = 0, ctas = 0;
        if ((e = batch_ctas_per_sm(&ctas)) != cudaSuccess) return e;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        max_warps = batch_warps(ctas, sms, a.num_tiles);
        if (max_warps == 0) {
            cfg = 2;  // the same 512-key tiles
            if ((e = range_max_warps(cfg, &max_warps)) != cudaSuccess) return e;
        }
    }
    if (!a.offsets || a.nseg < 1) return cudaErrorInvalidValue;
    return launch_mode<true, false>(dtype, incl, cfg, a, mi, mo, st, max_warps);
}

}  // namespace apsep
