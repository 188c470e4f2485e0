// apsep_internal.h -- layouts shared by the kernels and the C ABI.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "apsep.h"

namespace apsep {

// Error bits in Counters::err (read back by apsep_plan_check).
enum : uint32_t {
    ERR_LOOKBACK_TIMEOUT = 1u,  // a predecessor range never published
    ERR_TMA_TIMEOUT = 2u,       // a bulk copy did not complete in time
    ERR_INTERNAL = 4u,          // a search invariant failed (bug)
    ERR_BAD_OFFSETS = 8u,       // segment offsets not 0 = off[0] <= ... <= off[nseg] = n
};

// Look-back flag value (low 2 bits of a status word's tag).
constexpr uint32_t FLAG_AGG = 1u;
constexpr uint32_t EPOCH_LIMIT = (1u << 30) - 1u;

// Run-to-run control block at the head of a plan's scratch.  Zeroed once at
// creation with epoch = 1; each run leaves it ready for the next (the last
// CTA resets the counters and advances the epoch), so runs need no memset
// and can be captured in a CUDA graph.
struct alignas(64) Counters {
    uint32_t range_counter;  // next dynamic range id (one range per warp)
    uint32_t done;           // warps finished in the current run
    uint32_t epoch;          // tag of the current run's status words, 1..EPOCH_LIMIT
    uint32_t err;            // ERR_* bits, sticky until read
    uint32_t finished;       // ranges that published their minimum in the current run
    uint32_t pad[11];
};

// Scratch of one run, carved from one device allocation (or the static
// array of apsep_run_noalloc) by carve_scratch().
struct RangeScratch {
    Counters* ctr;
    uint64_t* group_min;    // [max_ranges/32] atomic min of (EPOCH_LIMIT - epoch) << 32 | ordered key
                            //   over each group of 32 ranges; all-ones when created
    uint64_t* range_state;  // [max_ranges] tag<<32 | key bits (4-byte keys): min of a finished range, for a
                            //   reader that waits on this word itself
    uint64_t* range_key;    // key[max_ranges] (packed): the range minima, for readers of the count too
    void* top_key;          // [max_ranges * kTopEntries] key: top of each range's final stack, bottom first
    int32_t* top_pos;       // [max_ranges * kTopEntries] their positions
    uint32_t* top_cnt;      // [max_ranges] entries published
    void* tile_min;         // [cap_tiles]  key: min of each tile
    void* chunk_min;        // [cap_chunks] key: min of each 32-key chunk
    uint32_t* tile_flag;    // [cap_tiles]  flagged keys of the tile | bit 31: some are capped
    uint32_t* tile_mask;    // [cap_tiles * kMaxTileKeys/32] which keys are flagged
    int cap_tiles;
    int max_ranges;
};

constexpr int kMinTileKeys = 256;   // smallest tile of any configuration (one warp's)
constexpr int kMaxTileKeys = 512;   // largest tile of any configuration
constexpr int kMaxRanges = 4096;    // persistent warps per run, upper bound
constexpr int kTopEntries = 32;           // stack entries each range publishes for later ranges

// Byte offsets of the scratch arrays for `capacity` keys (256-byte aligned).
struct ScratchOffsets {
    size_t gmin, state, rkey, topk, topp, topc, tmin, cmin, flag, mask, total;
    int64_t cap_tiles;
};
constexpr size_t align256(size_t x) { return (x + 255) / 256 * 256; }
// kb: bytes per key (4: int32 / float32; 8: int64 / float64).
constexpr ScratchOffsets scratch_offsets(int64_t capacity, int kb = 4) {
    ScratchOffsets o{};
    const int64_t cap = capacity > 0 ? capacity : 1;
    o.cap_tiles = (cap + kMinTileKeys - 1) / kMinTileKeys + 1;
    const size_t cap_chunks = (size_t)(cap + 31) / 32 + kMaxTileKeys / 32;
    o.gmin = align256(sizeof(Counters));
    o.state = align256(o.gmin + (size_t)(kMaxRanges / 32) * 8);
    o.rkey = align256(o.state + (size_t)kMaxRanges * 8);
    o.topk = align256(o.rkey + (size_t)kMaxRanges * 8);
    o.topp = align256(o.topk + (size_t)kMaxRanges * kTopEntries * kb);
    o.topc = align256(o.topp + (size_t)kMaxRanges * kTopEntries * 4);
    o.tmin = align256(o.topc + (size_t)kMaxRanges * 4);
    o.cmin = align256(o.tmin + (size_t)o.cap_tiles * kb);
    o.flag = align256(o.cmin + cap_chunks * kb);
    o.mask = align256(o.flag + (size_t)o.cap_tiles * 4);
    o.total = align256(o.mask + (size_t)o.cap_tiles * (kMaxTileKeys / 32) * 4);
    return o;
}

// The counters must start zeroed; a run leaves them zeroed, a run that timed
// out may not (apsep_plan_check clears them, keeping the epoch).
constexpr size_t control_bytes() { return sizeof(Counters); }
constexpr size_t group_min_bytes() { return (size_t)(kMaxRanges / 32) * 8; }

// Bytes of scratch for `capacity` keys of kb bytes; when base != nullptr also fills *s.
size_t carve_scratch(void* base, int64_t capacity, RangeScratch* s, int kb = 4);

#ifdef __CUDACC__
// Every kernel of the library is launched so that it may begin while the stream's
// previous kernel drains, and waits for that one's end and memory before its first
// global access: the launch itself (about 2 us between two dependent kernels) then
// overlaps (a run of 4000 keys 10.2 -> 8.0 us in a stream, 2^25 descending keys
// 58.6 -> 54.9).  A kernel that lets the next one start earlier, before its own
// end, gained nothing more.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchAttribute at[1] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}
#endif

struct RangeArgs {
    const void* d_in;
    int32_t* d_out;
    int n;
    int num_tiles;
    int tiles_per_range;
    int num_ranges;
    int tma_rows;            // floor(n/32): rows covered by the tensor maps (0 = no TMA)
    int head;                // 0..3 virtual keys in front of the array (d_in, d_out and n
                             //   include them) so that the TMA view starts 16-byte aligned;
                             //   never read or written, answers are relative to them
    uint32_t spin_limit;     // bound on every device-side wait (polls)
    int skip_publish_range;  // fault injection: this range never publishes (-1 = off)
    const int64_t* offsets;  // segmented runs: nseg + 1 segment offsets into d_in; else nullptr
    int nseg;
    RangeScratch s;
    int64_t* d_out64 = nullptr;  // int64 answers (the int64-position path's kernels): out_base + answer
    int64_t out_base = 0;
    int64_t unanswered64 = -1;  // what a key that no key of the run answers reads there
};

// Runs with int64 answers (RangeArgs::d_out64): a key that no key of the run
// answers reads RangeArgs::unanswered64 (UNRESOLVED64 when keys before the run may
// answer it, else -1), and a tile whose keys are all unanswered within
// their range is not written at all; its tile_flag word carries
// TILE_NOT_STORED (phase 2 still writes the keys that it answers).
constexpr int64_t UNRESOLVED64 = -2;
// Output forms of a run (the engine's OUTM template parameter): int32
// answers; int64 answers (above); int32 spans, position - answer.
constexpr int OUT_I32 = 0, OUT_I64 = 1, OUT_SPAN = 2;
constexpr uint32_t TILE_NOT_STORED = 0x40000000u;

// The TMA view of a run: the number of virtual keys (0..3) in front of d_in
// that put the view on a 16-byte boundary, or -1 when the input and the output
// sit at different offsets within 16 bytes (no common view: plain loads and
// stores throughout).  Tile 0, which holds the virtual keys, always takes the
// plain path, so nothing in front of the arrays is touched.
inline int view_head(const void* d_in, const void* d_out) {
    const int hi = (int)((uintptr_t)d_in % 16 / 4), ho = (int)((uintptr_t)d_out % 16 / 4);
    return hi == ho ? hi : -1;
}

// A kernel configuration: warps per CTA x keys per lane (a warp's tile is 32*ipt keys).
struct TileConfig {
    int wpc;
    int ipt;
};
constexpr int kNumTileConfigs = 6;
extern const TileConfig kTileConfigs[kNumTileConfigs];

// Launch one run.  Fills a.num_ranges / a.tiles_per_range from the
// configuration's occupancy on the current device.
cudaError_t launch_range(int dtype, int incl, int cfg, RangeArgs& a, const CUtensorMap& map_in,
                         const CUtensorMap& map_out, cudaStream_t stream);
cudaError_t range_prepare(int cfg);  // smem attributes + occupancy, current device
// Segmented runs (a.offsets, a.nseg set): the same engine, answers relative to
// each key's segment start.
cudaError_t launch_range_segmented(int dtype, int incl, int cfg, RangeArgs& a, const CUtensorMap& map_in,
                                   const CUtensorMap& map_out, cudaStream_t stream);
// 8-byte keys (dtype 2: int64, 3: float64), single arrays and segmented batches
// (RangeArgs::offsets): warp tiles of wide_tile_keys(...) keys, which the launch is
// given back (aligned: keys and answers on a 16-byte boundary); the int64-position path's pieces run in kWideTileKeys.
constexpr int kWideTileKeys = 256;
cudaError_t prepare_wide();
int wide_tile_keys(int64_t n, bool segmented, bool aligned);
cudaError_t launch_range_wide(int dtype, int incl, int tile_keys, RangeArgs& a, const CUtensorMap& map_in,
                              const CUtensorMap& map_out, cudaStream_t st);

// A single array behind a view head (RangeArgs::head > 0): the segmented
// kernel with one implicit segment and the whole-tile early paths.
cudaError_t prepare_view(int cfg, int* ctas_per_sm);
cudaError_t launch_range_view(int dtype, int incl, int cfg, RangeArgs& a, const CUtensorMap& map_in,
                              const CUtensorMap& map_out, cudaStream_t st);
cudaError_t prepare_segmented(int cfg, int* ctas_per_sm);
// Batches in configuration 0 have CTAs of their own, of kSegWarps warps.
constexpr int kSegWarps = 20;
// Persistent warps of such a batch of num_tiles tiles where ctas_per_sm of those
// CTAs are resident on each of sms SMs; 0: it takes configuration 2's kernel (fewer
// than six tiles a warp, measured in apsep_segmented.cu, or no CTA fits).
constexpr int batch_warps(int ctas_per_sm, int sms, int num_tiles) {
    const int w = ctas_per_sm * sms * kSegWarps < kMaxRanges ? ctas_per_sm * sms * kSegWarps : kMaxRanges;
    return w > 0 && num_tiles >= 6 * w ? w : 0;
}
cudaError_t batch_ctas_per_sm(int* ctas);  // their occupancy, current device (range_prepare(0))
cudaError_t range_max_warps(int cfg, int* warps);  // persistent warps of one launch, current device
// A single array (no view head) with int64 answers a.out_base + answer into
// a.d_out64 (4-byte keys in configuration 0, 8-byte keys in tiles of kWideTileKeys); flagged keys
// get a.unanswered64 and all-deferred tiles are not written (TILE_NOT_STORED).
cudaError_t launch_range_out64(int dtype, int incl, RangeArgs& a, const CUtensorMap& map_in, cudaStream_t st);
// A single array (no view head, 4-byte keys) through the order-reversing key
// map in configuration 0: previous-greater answers (int32), or with span != 0
// (strict comparison only) the stock span, position - answer.
cudaError_t launch_range_flipped(int dtype, int incl, int span, RangeArgs& a, const CUtensorMap& map_in,
                                 const CUtensorMap& map_out, cudaStream_t st);
// A single array (no view head, 4-byte keys) seen reversed in configuration
// 0: next-smaller answers (n - 1 - the reversed run's answer, at the mirrored
// position), TMA tiles only when n is a multiple of 32 (a.tma_rows * 32 == n).
cudaError_t launch_range_reversed(int dtype, int incl, RangeArgs& a, const CUtensorMap& map_in,
                                  const CUtensorMap& map_out, cudaStream_t st);
// The same two for 8-byte keys, in tiles of 512 (apsep_wide_mapped.cu).
constexpr int kWideMappedTileKeys = 512;
cudaError_t launch_wide_flipped(int dtype, int incl, int span, RangeArgs& a, const CUtensorMap& map_in,
                                const CUtensorMap& map_out, cudaStream_t st);
cudaError_t launch_wide_reversed(int dtype, int incl, RangeArgs& a, const CUtensorMap& map_in,
                                 const CUtensorMap& map_out, cudaStream_t st);
// Arms one-shot fault injection for the next apsep_run_noalloc call.
void noalloc_debug_inject(int32_t range, uint32_t spin_limit);

}  // namespace apsep

struct apsep_plan;
// One single-array run of the plan through the order-reversing key map
// (launch_range_flipped): previous greater (span = 0) or the stock span
// (span = 1, APSEP_LT).  APSEP_ENOTSUP when the engine has no such form for
// the call (8-byte keys in an array of short tiles, keys or answers off a 16-byte
// boundary, answers over the keys): the caller then takes its general route.
apsep_status plan_run_flipped(struct apsep_plan* plan, const void* d_in, int32_t* d_out, int64_t n, apsep_cmp cmp,
                              int span, void* stream);
// One single-array run of the plan over the reversed array
// (launch_range_reversed): out[i] = the next j > i with a[j] < a[i] (<= under
// APSEP_LE), else -1.  APSEP_ENOTSUP when the engine has no such form for the
// call (8-byte keys in an array of short tiles, keys or answers off a 16-byte
// boundary, n not a multiple of 32, answers over the keys): the caller then takes
// its general route.
apsep_status plan_run_reversed(struct apsep_plan* plan, const void* d_in, int32_t* d_out, int64_t n, apsep_cmp cmp,
                               void* stream);
// One single-array run of the plan with int64 answers (out_base + answer into
// d_out; see launch_range_out64): 4-byte keys in configuration 0, 8-byte keys
// in tiles of kWideTileKeys, by TMA when d_in is 16-byte aligned, else by plain loads.
// chunk_min, when not null, takes the run's minima of every 32 keys (in key
// order, up to the end of the last tile) instead of the plan's scratch.
// *layout returns the run's arguments: tile and range layout, scratch words.
apsep_status plan_run_out64(struct apsep_plan* plan, const void* d_in, int64_t* d_out, int64_t n, int64_t out_base,
                            apsep_cmp cmp, void* chunk_min, void* stream, apsep::RangeArgs* layout);
