// apsep_range_kernel.cuh -- the APSE engine for sm_103a: persistent,
// warp-independent ranges (single arrays and batches of segments).
//
// One launch.  Every WARP is an independent worker on a contiguous RANGE of
// warp tiles (32 lanes x IPT keys; the first warp of each CTA claims the
// CTA's consecutive ranges with one atomic, in CTA start order), with its own
// ring of TMA stages, its own answer buffers and its own stack in shared
// memory.  One __syncthreads publishes the claim; after it the warps
// synchronise only with __syncwarp.
//
//  Phase 1, per warp tile (the next tile's 128-byte-swizzled TMA load stays in
//  flight in the warp's ring):
//   1. whole-tile paths for sorted keys (single arrays);
//   2. in-thread answers over IPT consecutive keys in registers (compare
//      ladder) -- the in-thread step of apsepKernelSPT (src/apsep.cuh:2701-2707)
//      -- and, for a lane's first keys, over the four keys before the lane;
//   3. minima over lanes (src/apsep.cuh:2709-2730) and the tile's strict suffix
//      minima;
//   4. the keys left over, spread evenly over the lanes, find the nearest
//      earlier lane of the tile that qualifies by binary lifting over a 5-level
//      table of lane minima held in registers and their key by binary search
//      over that lane's suffix minima -- a fixed number of steps in place of
//      the reference's warp-uniform pointer jumping, spine walk and cross-warp
//      fallback (src/apsep.cuh:2734-2801);
//   5. keys without an answer in the tile search the warp's RANGE STACK (strict
//      suffix minima of the range's earlier tiles; its top 32 entries one per
//      lane, a shuffle search, binary search below), in place of the
//      reference's global min-tree descent (src/apsep.cuh:2952-2996) for every
//      answer inside the range; the rest are flagged for phase 2: deferred
//      (nothing in the range qualifies) or capped (the stack dropped the entry);
//   6. the whole tile leaves shared memory in one TMA store, flagged keys as
//      -1; the stack takes the tile's strict suffix minima.
//  Then the warp publishes its range minimum and the top of its stack, and
//  reads the exclusive prefix minimum P of the earlier ranges (one handshake
//  per launch, see range_publish).  Every wait is bounded and reports
//  ERR_LOOKBACK_TIMEOUT / ERR_TMA_TIMEOUT.
//
//  Phase 2 touches only the flagged keys.  Deferred keys are the range's
//  prefix minima, non-increasing, so the ones P qualifies form a prefix (the
//  reference's prefix-min early-out, src/apsep.cuh:2903-2926); each finds
//  the nearest earlier range whose minimum qualifies and its answer in that
//  range's published stack or its tile, chunk and key minima, 32 keys side by
//  side (answer_before); capped keys search their own range's tiles
//  (find_in_tiles).
//
//  On random keys the kernel is bound by the latency of its dependent steps
//  and by issue (4 warps a scheduler; 62 % of issue slots busy in the steady
//  state at 2^25 int32 keys): seeing four predecessors before any query,
//  one list and one prefix sum per tile, no prefix scan and one query round
//  took 2^25 uniform keys from 136 to 117 us and, with launches that overlap the
//  previous kernel and the shorter handshake, to 111 (2.4 TB/s of useful bytes);
//  the one-key-per-lane phase 2 with the longer stack and lists, and each stack top
//  copied once, took a random walk of 2^24 keys (stock span) from 783 to 140 us and
//  of 2^20 keys from 176 to 28.
#pragma once
#include "apsep_device.cuh"
#include "apsep_internal.h"

namespace apsep {

// TMA ring depth per warp (tiles): two, one landing while one is worked on (a
// third measured no gain for 4-byte keys, and its shared memory holds the longer
// stack and lists); three for 8-byte keys in tiles of 256 (ascending float64
// keys, 2^26 of them: 207 us with two, 173 us with three).
template <int KB, int IPT> constexpr int kStagesOf = KB == 8 && IPT == 8 ? 3 : 2;
// Range-stack entries kept per warp.  Random keys leave ~ln(range) suffix minima
// (10 of 13,800 keys), a random walk ~sqrt(range) (130): with 64 entries every
// second range of a walk dropped some and sent its keys to phase 2 as capped.
// (LEAN: the batches' 20-warp CTAs, whose shared memory leaves 128 entries.)
template <int KB, bool LEAN> constexpr int kStackCapOf = KB == 8 || LEAN ? 128 : 256;
constexpr int kUpKeep = 64;     // entries a wholly increasing tile leaves on the stack
constexpr int kXQueries = 3;    // cross-lane queries per lane and round (32 * 3 keys per round)
// Deferred keys listed in shared memory per range (a random walk's prefix
// minima, ~sqrt(range) of them, fit; 8-byte keys: what shared memory leaves).
template <int KB, int IPT, bool LEAN> constexpr int kDefCapOf = LEAN ? 64 : KB == 4 ? 192 : IPT == 8 ? 128 : 96;
constexpr int kCapCap = 32;     // capped keys listed in shared memory per range

// Shared memory of one warp (KB: bytes per key).
template <int IPT, int KB = 4, bool LEAN = false>
struct WLayout {
    static constexpr int WT = 32 * IPT;                              // keys per warp tile
    static constexpr size_t kV = 0;                                   // T[S][WT], swizzled (TMA dst)
    static constexpr size_t kO = kV + (size_t)kStagesOf<KB, IPT> * WT * KB;      // int32[WT], swizzled (TMA src)
    static constexpr size_t kSM = kO + (size_t)WT * 4;                // T[WT], swizzled: lane suffix minima
    static constexpr size_t kList = kSM + (size_t)WT * KB;            // int16[WT]: X keys in order
    static constexpr size_t kStkV = kList + (size_t)WT * 2;           // T[K]
    static constexpr size_t kStkP = kStkV + (size_t)kStackCapOf<KB, LEAN> * KB;   // int32[K]
    static constexpr size_t kDefP = kStkP + (size_t)kStackCapOf<KB, LEAN> * 4;    // int32[kDefCap]
    static constexpr size_t kDefV = kDefP + (size_t)kDefCapOf<KB, IPT, LEAN> * 4;  // T[kDefCap]
    static constexpr size_t kCapP = kDefV + (size_t)kDefCapOf<KB, IPT, LEAN> * KB;  // int32[kCapCap]
    static constexpr size_t kCapS = kCapP + (size_t)kCapCap * 4;      // int32[kCapCap]: segment starts
    static constexpr size_t kPad = (kCapS + (size_t)kCapCap * 4 + 15) / 16 * 16;  // T[4]: pads (lane 0's earlier keys)
    static constexpr size_t kBar = kPad + 4 * KB;  // uint64[S]
    static constexpr size_t kFlag = kBar + (size_t)kStagesOf<KB, IPT> * 8;  // int32: phase 2's group minima are staged
    static constexpr size_t kEnd = kFlag + 8;
    static constexpr size_t kBytes = (kEnd + 1023) / 1024 * 1024;     // keeps every warp 1024-aligned
    static_assert(kO % 1024 == 0 && kSM % 1024 == 0 && (WT * KB) % 1024 == 0,
                  "swizzled buffers need 1024-byte alignment");
    static_assert(kStkV % 8 == 0 && kDefV % 8 == 0, "8-byte keys need 8-byte aligned arrays");
};

template <int IPT, int WPC, int KB = 4, bool LEAN = false>
constexpr size_t kernel_smem_bytes() { return WLayout<IPT, KB, LEAN>::kBytes * WPC + 1024 + 64; }  // + CTA words

// Key of a group word (the low half of an atomic minimum over ordered keys).
template <typename T>
__device__ __forceinline__ T group_key(const uint64_t* w) {
    return KeyTraits<T>::from_ord((uint32_t)__ldcg((const unsigned long long*)w));
}

// The published minimum of range i: the word that the publication releases
// (range_publish).  Not the tagged word: that one is only for a reader that
// acquires it itself.
template <typename T>
__device__ __forceinline__ T range_min(const RangeArgs& a, int i) {
    return __ldcg((const T*)a.s.range_key + i);
}

// The minimum of group g (32 ranges), every range of which has published:
// its atomic word for 4-byte keys, the minimum of its ranges' words for
// 8-byte keys (no 64-bit key fits beside a tag in one atomic word).
template <typename T>
__device__ __forceinline__ T group_min_of(const RangeArgs& a, int g) {
    if constexpr (sizeof(T) == 8) {
        const ulonglong2* w = reinterpret_cast<const ulonglong2*>(&a.s.range_key[32 * g]);
        ulonglong2 u[16];  // every range of the group is there: it lies before some published range's group
#pragma unroll
        for (int i = 0; i < 16; i++) u[i] = __ldcg(w + i);
        T m = KeyTraits<T>::pad();
#pragma unroll
        for (int i = 0; i < 16; i++)
            m = KeyTraits<T>::vmin(m, KeyTraits<T>::vmin(KeyTraits<T>::from_bits((uint64_t)u[i].x),
                                                         KeyTraits<T>::from_bits((uint64_t)u[i].y)));
        return m;
    } else {
        return group_key<T>(&a.s.group_min[g]);
    }
}

// Exclusive prefix sum over the warp's lanes of a count c, and the total.
__device__ __forceinline__ int warp_excl_sum(int c, int& total) {
    int x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int nb = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)(threadIdx.x & 31) >= o) x += nb;
    }
    total = __shfl_sync(0xffffffffu, x, 31);
    return x - c;
}

// Segmented runs: the segment holding position pos -- the largest s < nseg
// with off[s] <= pos (off[0] = 0 <= pos).  Warp-cooperative, 32 candidates
// per step, so about log32(nseg) dependent reads.
static __device__ __noinline__ int seg_find(const int64_t* __restrict__ off, int nseg, int pos, uint32_t* err) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = nseg;
    while (true) {
        const int step = hi - lo > 32 ? (hi - lo + 31) / 32 : 1;
        const int idx = lo + lane * step;
        const bool ok = idx < hi && __ldg(&off[idx]) <= (int64_t)pos;
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if (!m) {  // offsets not as promised (off[lo] > pos); stay in bounds
            if (lane == 0) atomicOr(err, ERR_BAD_OFFSETS);
            return lo;
        }
        lo += (31 - __clz(m)) * step;
        if (step == 1) return lo;
        hi = min(lo + step, hi);
    }
}

// Answer relative to the segment start s: an answer before the segment is none.
__device__ __forceinline__ int seg_rel(int g, int s) { return g >= s ? g - s : -1; }

// The key at position pos of the run's array, through the key map; REV runs
// see the array reversed (position pos is element n - 1 - pos).
template <typename T, int KMAP, bool REV>
__device__ __forceinline__ T key_at(const T* d_in, int n, int pos) {
    return load_key<T, KMAP>(d_in + (REV ? n - 1 - pos : pos));
}

// N consecutive keys or minima through L2, 16 bytes per load where they are aligned.
template <typename T, int N>
__device__ __forceinline__ void load_run(const T* p, T (&m)[32]) {
    constexpr int PER = 16 / (int)sizeof(T);
    static_assert(N <= 32 && N % PER == 0, "whole 16-byte loads");
    if (((uintptr_t)p & 15) == 0) {
        uint4 w[N / PER];
#pragma unroll
        for (int k = 0; k < N / PER; k++) w[k] = __ldcg(reinterpret_cast<const uint4*>(p) + k);
#pragma unroll
        for (int k = 0; k < N / PER; k++) {
            if constexpr (sizeof(T) == 4) {
                m[4 * k] = KeyTraits<T>::from_bits(w[k].x);
                m[4 * k + 1] = KeyTraits<T>::from_bits(w[k].y);
                m[4 * k + 2] = KeyTraits<T>::from_bits(w[k].z);
                m[4 * k + 3] = KeyTraits<T>::from_bits(w[k].w);
            } else {
                m[2 * k] = KeyTraits<T>::from_bits(((uint64_t)w[k].y << 32) | w[k].x);
                m[2 * k + 1] = KeyTraits<T>::from_bits(((uint64_t)w[k].w << 32) | w[k].z);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; k++) m[k] = __ldcg(p + k);
    }
}

// Phase 2's searches take up to kFew queries one by one, the warp's lanes side by
// side on 32 entries of a level (one load and a ballot a step), and more of them
// one per lane (a round of independent loads a step for all): a lone query is
// three times slower the second way, 32 of them ten times slower the first.
constexpr int kFew = 4;

// The last of the entries lo..hi (hi - lo < 32) that qualifies, or -1; uniform call.
template <typename T, bool INCL, typename Load>
__device__ __forceinline__ int last_of(int lo, int hi, T q, Load load) {
    const int i = hi - (int)(threadIdx.x & 31);
    const unsigned m = __ballot_sync(0xffffffffu, i >= lo && lt<INCL>(load(max(i, lo)), q));
    return m ? hi - (__ffs(m) - 1) : -1;
}

// Search inside one range: each lane with `need` finds the rightmost key that
// qualifies for its q in its tiles [lo, hi) -- the nearest tile by tile minima,
// its chunk, its key.  -2 when no tile's minimum qualifies; exact = false: some
// tile's minimum is known to qualify.
template <typename T, int B, bool INCL, int MAPF = KMAP_NONE, bool REV = false>
__device__ __noinline__ int find_in_tiles(T q, bool need, int lo, int hi, bool exact, const T* __restrict__ d_in,
                                          const RangeArgs& a) {
    constexpr int W = B / 32;
    const T* tile_min = (const T*)a.s.tile_min;
    const T* chunk_min = (const T*)a.s.chunk_min;
    unsigned nm = __ballot_sync(0xffffffffu, need);
    if (__popc(nm) <= kFew) {
        int p = -2;
        for (; nm; nm &= nm - 1) {
            const int f = __ffs(nm) - 1;
            const T qf = __shfl_sync(0xffffffffu, q, f);
            const int lf = __shfl_sync(0xffffffffu, lo, f), hf = __shfl_sync(0xffffffffu, hi, f);
            int s = -1;
            for (int h = hf - 1; h >= lf && s < 0; h -= 32)
                s = last_of<T, INCL>(max(lf, h - 31), h, qf, [&](int i) { return __ldcg(&tile_min[i]); });
            if (s < 0) continue;
            const int c = max(last_of<T, INCL>(0, W - 1, qf, [&](int i) { return __ldcg(&chunk_min[(size_t)s * W + i]); }), 0);
            const int row = s * B + c * 32;
            const int k = last_of<T, INCL>(max(row, a.head), row + 31, qf,
                                           [&](int i) { return key_at<T, MAPF, REV>(d_in, a.n, min(i, a.n - 1)); });
            if ((int)(threadIdx.x & 31) == f && k >= 0 && k < a.n) p = k;
        }
        return p;
    }
    int s = hi - lo == 1 && !exact ? lo : -1;  // (a range of one tile whose minimum is known to qualify)
    for (int t = hi - 1; need && s < 0 && t >= lo; t -= 16) {
        T m[16];
#pragma unroll
        for (int k = 0; k < 16; k++) m[k] = t - k >= lo ? __ldcg(&tile_min[t - k]) : KeyTraits<T>::pad();
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (s < 0 && t - k >= lo && lt<INCL>(m[k], q)) s = t - k;
    }
    int p = -2;
    if (need && s >= 0) {
        T m[32];
        load_run<T, W>(chunk_min + (size_t)s * W, m);
        int c = 0;
#pragma unroll
        for (int k = 0; k < W; k++)
            if (lt<INCL>(m[k], q)) c = k;
        const int row = s * B + c * 32;  // (whole tiles lie below hi: the row ends inside the array)
        if (row >= a.head) {
            load_run<T, 32>(d_in + (REV ? a.n - 32 - row : row), m);
        } else {  // the view's virtual keys are not read
#pragma unroll
            for (int k = 0; k < 32; k++) m[k] = __ldcg(&d_in[max(row + k, a.head)]);
        }
#pragma unroll
        for (int k = 0; k < 32; k++)
            if (row + k >= a.head && lt<INCL>(map_key<T, MAPF>(m[REV ? 31 - k : k]), q)) p = row + k;
    }
    __syncwarp();
    return p;
}

// Phase 2: each lane with `want` finds the answer of its q before range r (the
// prefix minimum of the earlier ranges qualifies for it): the
// nearest range whose minimum qualifies -- by the window of 32 range minima
// (lane i: range r-1-i; wpm: their running minimum), else by the running minima
// of the earlier groups (sg, staged in shared memory at the first need) and
// that group's 32 range minima -- then the topmost qualifying entry of that
// range's published stack, else its tiles.  -2: the published minima contradict
// each other.
template <typename T, int B, bool INCL, int MAPF = KMAP_NONE, bool REV = false>
__device__ __noinline__ int answer_before(T q, bool want, int r, T wpm, T* sg, int* staged,
                                          const T* __restrict__ d_in, const RangeArgs& a) {
    constexpr unsigned FULL = 0xffffffffu;
    constexpr int KB = (int)sizeof(T);
    const int lane = threadIdx.x & 31;
    int rp = -1;
    {
        int lo = -1;  // the nearest lo + 1 ranges do not qualify
#pragma unroll 1
        for (int s = 16; s > 0; s >>= 1)
            if (!lt<INCL>(__shfl_sync(FULL, wpm, lo + s), q)) lo += s;
        if (lt<INCL>(__shfl_sync(FULL, wpm, lo + 1), q)) rp = max(r - 2 - lo, -1);
    }
    unsigned far = __ballot_sync(FULL, want && rp < 0);  // answers before the window
    if (__popc(far) <= kFew) {
        for (; far; far &= far - 1) {
            const int f = __ffs(far) - 1;
            const T qf = __shfl_sync(FULL, q, f);
            int rf = -1;
            if constexpr (KB == 8) {  // no group words: the range minima, 8 groups a step
                for (int hi = r - 33; hi >= 0 && rf < 0; hi -= 256) {
                    T u[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) u[k] = range_min<T>(a, max(hi - 32 * k - lane, 0));
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const unsigned b = __ballot_sync(FULL, hi - 32 * k - lane >= 0 && lt<INCL>(u[k], qf));
                        if (b && rf < 0) rf = hi - 32 * k - (__ffs(b) - 1);
                    }
                }
            } else {
                int gf = -1;
                for (int g = r < 33 ? -1 : (r - 33) >> 5; g >= 0 && gf < 0; g -= 32)
                    gf = last_of<T, INCL>(max(g - 31, 0), g, qf, [&](int i) { return group_min_of<T>(a, i); });
                if (gf >= 0) rf = last_of<T, INCL>(32 * gf, 32 * gf + 31, qf, [&](int i) { return range_min<T>(a, i); });
            }
            if (lane == f) rp = rf;
        }
    } else {
        const int ng = r >= 33 ? ((r - 33) >> 5) + 1 : 0;  // groups of earlier ranges (the window's part does not qualify)
        static_assert(kMaxRanges / 32 == 128, "four groups per lane");
        if (!*staged) {
            __syncwarp();
#pragma unroll 1
            for (int g = lane; g < kMaxRanges / 32; g += 32) {
                T m = KeyTraits<T>::pad();
                if (g < ng) m = group_min_of<T>(a, g);
                sg[g] = m;
            }
            __syncwarp();
            T m[4];
#pragma unroll
            for (int j = 0; j < 4; j++) m[j] = sg[4 * lane + j];
#pragma unroll
            for (int j = 2; j >= 0; j--) m[j] = KeyTraits<T>::vmin(m[j], m[j + 1]);
            T x = m[0];
#pragma unroll 1
            for (int o = 1; o < 32; o <<= 1) {
                const T y = __shfl_down_sync(FULL, x, o);
                if (lane + o < 32) x = KeyTraits<T>::vmin(x, y);
            }
            const T after = __shfl_down_sync(FULL, x, 1);
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; j++) sg[4 * lane + j] = lane < 31 ? KeyTraits<T>::vmin(m[j], after) : m[j];
            if (lane == 0) *staged = 1;
            __syncwarp();
        }
        if (want && rp < 0 && ng > 0) {
            int g = 0;
#pragma unroll 1
            for (int s = 64; s > 0; s >>= 1)
                if (g + s < ng && lt<INCL>(sg[g + s], q)) g += s;
            T m[32];  // its 32 range minima
            load_run<T, 32>((const T*)a.s.range_key + 32 * g, m);
#pragma unroll
            for (int k = 0; k < 32; k++)
                if (lt<INCL>(m[k], q)) rp = 32 * g + k;
        }
    }
    // The published stack tops of the ranges that lanes ask for, up to kSlots of them
    // copied to shared memory at a time, each by the first lane that asks for it (all
    // copies in flight together), then searched by the lanes side by side: entries
    // increase from the bottom, so the qualifying ones form a bottom part and the
    // topmost of them answers.
    using L = WLayout<B / 32, KB>;
    constexpr int kRoom = (int)((L::kList - L::kV - KB * (kMaxRanges / 32)) / (32 * (KB + 4)));
    constexpr int kSlots = kRoom < 16 ? kRoom : 16;
    static_assert(kSlots >= 8, "room for phase 2's staging");
    static_assert(kTopEntries == 32, "a lane copies 2 KB + 8 times 16 bytes");
    T* sk = sg + kMaxRanges / 32;               // T[kSlots][32]
    int32_t* sp = (int32_t*)(sk + kSlots * 32);  // int32[kSlots][32]
    int ans = -2;
    const int rq = want ? rp : -1;
    const int first = __ffs(__match_any_sync(FULL, rq)) - 1;  // the first lane with this lane's range
    const unsigned firsts = __ballot_sync(FULL, rq >= 0 && first == lane);
    const int nth = __popc(firsts & ((1u << first) - 1u));
    for (int s0 = 0; s0 < __popc(firsts); s0 += kSlots) {
        const int slot = rq >= 0 ? nth - s0 : -1;
        int cnt = 0;
        __syncwarp();
        if (slot >= 0 && slot < kSlots && first == lane) {
            cnt = (int)__ldcg(&a.s.top_cnt[rq]);
            const char* tk = (const char*)((const T*)a.s.top_key + (size_t)rq * kTopEntries);
            const char* tp = (const char*)(a.s.top_pos + (size_t)rq * kTopEntries);
#pragma unroll
            for (int k = 0; k < 2 * KB; k++) copy_async16((char*)(sk + slot * 32) + 16 * k, tk + 16 * k);
#pragma unroll
            for (int k = 0; k < 8; k++) copy_async16((char*)(sp + slot * 32) + 16 * k, tp + 16 * k);
        }
        copy_async_wait();
        __syncwarp();
        cnt = __shfl_sync(FULL, cnt, first);
        if (slot >= 0 && slot < kSlots) {
            int lo = -1;
#pragma unroll 1
            for (int s = 32; s > 0; s >>= 1)
                if (lo + s < cnt && lt<INCL>(sk[slot * 32 + lo + s], q)) lo += s;
            if (lo >= 0) ans = sp[slot * 32 + lo];
        }
    }
    const bool miss = want && rp >= 0 && ans == -2;
    if (__any_sync(FULL, miss)) {
        const int lo = max(rp, 0) * a.tiles_per_range;
        const int found =
            find_in_tiles<T, B, INCL, MAPF, REV>(q, miss, lo, min(lo + a.tiles_per_range, a.num_tiles), false, d_in, a);
        if (miss) ans = found;
    }
    return ans;
}

// ---------------------------------------------------------------------------
// Range minima -> exclusive prefix minima.
//
// Publishing range r (lane 0): its minimum (range_key), an atomic minimum into
// its group's word (groups of 32 ranges; 4-byte keys), a fence, then the range's
// tagged word (range_state) and one fire-and-forget increment of the count of
// published ranges.  The one fence releases everything before it, both to a reader
// of the tagged word and to a reader of the count; nothing orders those two stores,
// so a reader of the count reads only what lies before the fence (the minimum's
// own store is free: 2^25 uniform int32 keys 111.3 us with it, 111.3 when the minima
// were read from the tagged words).  One
// warp per CTA polls that count (152 pollers), the others a word in shared
// memory.  Range r then needs the minima of the earlier ranges of its group
// plus those of the earlier groups: one round of loads, and no step of the last
// range's path waits on another range's loads.  (With the last range raising a
// flag per CTA, two more fences and a store and a load through L2, a run took
// 0.6-1.4 us longer: 2^18 uniform keys 14.2 -> 12.9 us.  One warp loading the
// minima for its whole CTA took 1 us longer again.)
//
// Group words: atomic minima of (EPOCH_LIMIT - epoch) << 32 | ordered key.
// The current run's tag is below every older run's, so its first minimum
// replaces an older word and the words need no reset between runs (they
// start all-ones and are cleared again when the epoch wraps).
//
// Every range of a launch is resident when the launch fits the device (the
// grid is sized from occupancy), so the count always completes.  When it does
// not within a bound (the launch shares the device and some warps
// have not started), range r falls back to waiting on the tagged minima of
// the ranges before it, all of which already run (ids are handed out in
// start order), so no wait depends on a warp that may not start.  Every wait
// is bounded and reports ERR_LOOKBACK_TIMEOUT when it gives up.
// ---------------------------------------------------------------------------
// A launch of at most kDirectRanges ranges skips the count: range r polls
// the tagged minima of the ranges before it directly (two words a lane), which ends
// sooner than waiting for every range of the launch to publish (32 ranges 7.9
// against 8.9 us a run, 64 ranges 8.7 against 9.5); with 256 ranges the pollers'
// own traffic costs more (12.3 against 10.2 us).
constexpr int kDirectRanges = 64;

template <typename T>
__device__ void range_publish(int r, uint32_t epoch, T rmin, const RangeArgs& a) {
    const uint32_t tag = (epoch << 2) | FLAG_AGG;
    if ((threadIdx.x & 31) == 0 && r != a.skip_publish_range) {
        __stcg((T*)a.s.range_key + r, rmin);
        if constexpr (sizeof(T) == 4)
            red_min_u64(&a.s.group_min[r >> 5], ((uint64_t)(EPOCH_LIMIT - epoch) << 32) | KeyTraits<T>::ord(rmin));
        // release: this range's words (every lane's, ordered by the caller's
        // __syncwarp), its minimum and the group's before the tagged word and the count
        fence_acq_rel();
        __stcg((unsigned long long*)&a.s.range_state[r],
               ((uint64_t)tag << 32) | (sizeof(T) == 8 ? 0u : (uint32_t)KeyTraits<T>::bits(rmin)));
        if (a.num_ranges > kDirectRanges) red_add_u32(&a.s.ctr->finished, 1u);
    }
}

// p: the minimum over ranges [0, r); win (lane i): the minimum of range r-1-i
// (pad below range 0), the window phase 2 searches first.  has_p: there is a p (not
// in range 0, nor when the wait gave up).
template <typename T>
__device__ void range_prefix(int r, uint32_t epoch, const RangeArgs& a, int* sReady, T& p, bool& has_p, T& win) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int g = r >> 5;
    const uint32_t tag = (epoch << 2) | FLAG_AGG;
    p = KeyTraits<T>::pad();
    win = KeyTraits<T>::pad();
    has_p = r > 0;
    if (r == 0) return;
    const uint32_t* count = &a.s.ctr->finished;
    const uint32_t all = (uint32_t)a.num_ranges;
    // every range has published: the window (it holds the group's earlier
    // ranges) and the earlier groups, in one round of loads
    auto from_ready = [&]() {
        const int wi = r - 1 - lane;
        win = wi >= 0 ? range_min<T>(a, wi) : KeyTraits<T>::pad();
        T m = wi >= g * 32 ? win : KeyTraits<T>::pad();
        if constexpr (sizeof(T) == 8) {  // the ranges of the earlier groups, one by one
            for (int i = lane; i < g * 32; i += 32) m = KeyTraits<T>::vmin(m, range_min<T>(a, i));
        } else {
            const uint32_t gtag = EPOCH_LIMIT - epoch;
            bool bad = false;
#pragma unroll
            for (int k = 0; k < kMaxRanges / 32 / 32; k++) {
                const int gi = lane + 32 * k;
                if (gi < g) {
                    const uint64_t w = __ldcg((const unsigned long long*)&a.s.group_min[gi]);
                    bad = bad || (uint32_t)(w >> 32) != gtag;
                    m = KeyTraits<T>::vmin(m, KeyTraits<T>::from_ord((uint32_t)w));
                }
            }
            if (bad) atomicOr(&a.s.ctr->err, ERR_INTERNAL);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = KeyTraits<T>::vmin(m, __shfl_xor_sync(FULL, m, o));
        p = m;
    };
    // 1. the count of published ranges, polled by the first warp of the CTA that gets
    //    here; the others watch its word in shared memory (0: waiting, 1: every
    //    range has published, 2: gave up).  A launch of few ranges has no count: its
    //    ranges wait on their predecessors.
    int ready = 0;
    if (lane == 0 && a.num_ranges > kDirectRanges) {
        const uint32_t bound = min(a.spin_limit, 1u << 16);
        volatile int* word = sReady;
        if (atomicExch(sReady + 1, 1) == 0) {
            for (uint32_t s = 0;; s++) {
                if (ld_acquire_u32(count) == all) {
                    ready = 1;
                    break;
                }
                if (s >= bound) break;
                if (s >= 64) __nanosleep(64);
            }
            __threadfence_block();
            *word = ready ? 1 : 2;
        } else {
            int w;
            for (uint32_t s = 0; (w = *word) == 0 && s < 16 * bound; s++) __nanosleep(32);
            __threadfence_block();
            ready = w == 1;
        }
    }
    __syncwarp();  // lane 0's acquire before the other lanes' loads
    if (__shfl_sync(FULL, ready, 0)) {
        from_ready();
        return;
    }
    // 2. fallback: wait for the tagged minima of the earlier ranges (or the count)
    for (uint32_t spins = 0;; spins++) {
        bool ok = true;
        T m = KeyTraits<T>::pad();
        for (int ri = lane; ri < r; ri += 32) {
            const uint64_t w = ld_acquire_u64(&a.s.range_state[ri]);
            if ((uint32_t)(w >> 32) != tag) ok = false;
            m = KeyTraits<T>::vmin(m, sizeof(T) == 8 ? range_min<T>(a, ri) : KeyTraits<T>::from_bits((uint32_t)w));
        }
        if (__all_sync(FULL, ok)) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = KeyTraits<T>::vmin(m, __shfl_xor_sync(FULL, m, o));
            p = m;
            __syncwarp();  // the window's ranges are ones that other lanes acquired (a vote orders nothing)
            const int wi = r - 1 - lane;
            win = wi >= 0 ? range_min<T>(a, wi) : KeyTraits<T>::pad();
            return;
        }
        if (__shfl_sync(FULL, lane == 0 && a.num_ranges > kDirectRanges ? (int)(ld_acquire_u32(count) == all) : 0, 0)) {
            __syncwarp();
            from_ready();
            return;
        }
        if (spins >= a.spin_limit) {
            if (lane == 0) atomicOr(&a.s.ctr->err, ERR_LOOKBACK_TIMEOUT);
            has_p = false;  // what those ranges would publish may be an older run's: phase 2 leaves it alone
            return;
        }
        __nanosleep(spins < 128 ? 64 : 256);
    }
}

// ---------------------------------------------------------------------------
// Phase 2 of range r: its flagged keys, whose answers need the other ranges'
// publications.  A function of its own: its registers (up to 32 loads in flight a
// lane) then cost phase 1 none (inlined, the 8-byte kernels spilled there: 125 ->
// 142 us at 2^24 int64 keys).
// ---------------------------------------------------------------------------
template <typename T, int IPT, bool INCL, bool SEG, bool LEAN, int MAPF, int OUTM, bool REV>
__device__ __noinline__ void phase2(const RangeArgs& a, unsigned char* wsm, const int r, const int t0, const int t1,
                                    const int def_total, const int cap_total, const int first_start, const T P,
                                    const bool has_p, const T win) {
    constexpr int KB = (int)sizeof(T);
    using L = WLayout<IPT, KB, LEAN>;
    constexpr int WT = L::WT, W = WT / 32, RPT = W * KB / 4, MW = kMaxTileKeys / 32, kDefCap = kDefCapOf<KB, IPT, LEAN>;
    constexpr unsigned FULL = 0xffffffffu;
    constexpr bool OUT64 = OUTM == OUT_I64;
    const int lane = threadIdx.x & 31;
    T* sV = (T*)(wsm + L::kV);
    int16_t* sList = (int16_t*)(wsm + L::kList);
    const int32_t* sDefP = (const int32_t*)(wsm + L::kDefP);
    const T* sDefV = (const T*)(wsm + L::kDefV);
    const int32_t* sCapP = (const int32_t*)(wsm + L::kCapP);
    const int32_t* sCapS = (const int32_t*)(wsm + L::kCapS);
    const T* d_in = (const T*)a.d_in;
    uint32_t* err = &a.s.ctr->err;
    const int head = SEG ? a.head : 0;
    auto seg_off = [&](int i) -> int64_t {
        return a.offsets ? (int64_t)__ldg(&a.offsets[i]) : (i == 0 ? (int64_t)0 : (int64_t)(a.n - head));
    };
    auto seg_idx = [&](int pos) { return a.offsets ? seg_find(a.offsets, a.nseg, pos, err) : 0; };
    auto tile_full = [&](int t) { return a.tma_rows > 0 && (t + 1) * RPT <= a.tma_rows && (t > 0 || head == 0); };
    // a final answer v of position pos (phase 2); int64 answers: out_base + v, and
    // a.unanswered64 for none (the int64-position path's mark); spans:
    // pos - v
    auto put = [&](int pos, int v) {
        if constexpr (OUT64) a.d_out64[pos] = v >= 0 ? (int64_t)v + a.out_base : a.unanswered64;
        else if constexpr (REV) a.d_out[a.n - 1 - pos] = v >= 0 ? a.n - 1 - v : -1;
        else if constexpr (OUTM == OUT_SPAN) a.d_out[pos] = pos - v;
        else a.d_out[pos] = v;
    };
    // the same for the four positions from pos on (a multiple of 4, in a tile that
    // streams through TMA: 16-byte aligned), v >= 0
    auto put4 = [&](int pos, int v) {
        if constexpr (OUT64) {
            const long long w = (long long)v + a.out_base;
            longlong2* o = reinterpret_cast<longlong2*>(a.d_out64 + pos);
            if (((uintptr_t)o & 15) == 0) {
                o[0] = make_longlong2(w, w);
                o[1] = make_longlong2(w, w);
            } else {
                for (int k = 0; k < 4; k++) a.d_out64[pos + k] = w;
            }
        } else if constexpr (REV) {
            const int w = a.n - 1 - v;
            *reinterpret_cast<int4*>(a.d_out + (a.n - 4 - pos)) = make_int4(w, w, w, w);
        } else if constexpr (OUTM == OUT_SPAN) {
            *reinterpret_cast<int4*>(a.d_out + pos) = make_int4(pos - v, pos + 1 - v, pos + 2 - v, pos + 3 - v);
        } else {
            *reinterpret_cast<int4*>(a.d_out + pos) = make_int4(v, v, v, v);
        }
    };

    // ======================= phase 2: flagged keys ===============================
    const int range_begin = t0 * WT;
    T* sg = sV;  // the TMA ring is idle now: running minima of the earlier groups
    int* staged = (int*)(wsm + L::kFlag);
    if (lane == 0) *staged = 0;
    __syncwarp();
    T wpm = win;  // running minima of the window, from the nearest range on
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T nb = __shfl_up_sync(FULL, wpm, o);
        if (lane >= o) wpm = KeyTraits<T>::vmin(wpm, nb);
    }

    // A. deferred keys: the range's prefix minima, non-increasing, so the ones P
    //    qualifies form a prefix of them and the rest keep -1.  Answers of
    //    non-increasing queries only move left, so while the last answer's key
    //    (the cursor) still qualifies it is the answer; else answer_before,
    //    one key per lane.
    bool a_done = !has_p;
    int cur = -1;
    T cv = KeyTraits<T>::pad();
    // up to 32 deferred keys in order, one per lane (uniform call)
    auto deferred32 = [&](const bool in, const T q, const int pos) {
        const bool want = in && lt<INCL>(P, q);  // (segmented: all of the range's first segment)
        if (__ballot_sync(FULL, want) != __ballot_sync(FULL, in)) a_done = true;
        const bool ok = want && cur >= 0 && lt<INCL>(cv, q);
        if (ok && (!head || pos >= head)) put(pos, SEG ? seg_rel(cur, first_start) : cur);
        const bool rest = want && !ok;
        const unsigned rm = __ballot_sync(FULL, rest);
        if (!rm) return;
        const int ans = answer_before<T, WT, INCL, MAPF, REV>(q, rest, r, wpm, sg, staged, d_in, a);
        if (rest) {
            if (ans < 0) atomicOr(err, ERR_INTERNAL);
            else if (!head || pos >= head) put(pos, SEG ? seg_rel(ans, first_start) : ans);
        }
        cur = __shfl_sync(FULL, ans, 31 - __clz(rm));
        if (cur < 0) {
            a_done = true;
        } else if (SEG && cur < first_start) {
            a_done = true;  // before the segment: so are the answers of the lower keys (-1 already)
        } else if (!a_done) {
            cv = key_at<T, MAPF, REV>(d_in, a.n, cur);
        }
    };
    const int nlist = min(def_total, kDefCap);
    for (int b0 = 0; b0 < nlist && !a_done; b0 += 32) {
        const int j = b0 + lane;
        const bool in = j < nlist;
        deferred32(in, in ? sDefV[j] : KeyTraits<T>::pad(), in ? sDefP[j] : 0);
    }
    // The flagged keys at or after `from` of tile t, 32 per step (uniform call).  A
    // mixed tile's keys look in the earlier tiles of the range first (capped keys
    // are answered there, deferred ones are not); with_deferred: keys without an
    // answer there go to deferred32.
    auto flagged_tile = [&](const int t, const bool mixed, const int from, const bool with_deferred) {
        uint32_t mw = lane < W ? __ldcg(&a.s.tile_mask[(size_t)t * MW + lane]) : 0u;
        if (lane < W) {
            const int p0 = t * WT + 32 * lane, lim = max(from, head);
            if (p0 < lim) mw &= lim - p0 >= 32 ? 0u : (0xffffffffu << (lim - p0));
        }
        int tot;
        int off = warp_excl_sum(__popc(mw), tot);
        __syncwarp();
        while (mw) {
            const int k = __ffs(mw) - 1;
            mw &= mw - 1;
            sList[off++] = (int16_t)(32 * lane + k);
        }
        __syncwarp();
        for (int b0 = 0; b0 < tot; b0 += 32) {
            bool in = b0 + lane < tot;
            const int pos = t * WT + (in ? (int)sList[b0 + lane] : 0);
            const T q = in ? key_at<T, MAPF, REV>(d_in, a.n, pos) : KeyTraits<T>::pad();
            if (mixed) {
                const int found = find_in_tiles<T, WT, INCL, MAPF, REV>(q, in, t0, t, true, d_in, a);
                if constexpr (SEG) {  // the keys' own segments, one after another
                    for (unsigned m = __ballot_sync(FULL, in && found >= 0); m; m &= m - 1) {
                        const int f = __ffs(m) - 1;
                        const int sf = (int)seg_off(seg_idx(__shfl_sync(FULL, pos, f) - head)) + head;
                        if (lane == f) put(pos, seg_rel(found, sf));
                    }
                } else if (in && found >= 0) {
                    put(pos, found);
                }
                // (segmented: flagged keys without an answer in the range are of its first segment)
                in = in && found < 0;
            }
            if (with_deferred && !a_done) deferred32(in, q, pos);
        }
        __syncwarp();
    };
    if (!a_done && def_total > kDefCap) {
        // A'. the list overflowed and P qualified every listed key: continue over
        //     the tile flags after the last listed key, 32 tiles per load.
        const int from = sDefP[kDefCap - 1] + 1;
        constexpr int TPL = 32 / W;  // tiles per load of mask words
        const T* tile_min_r = (const T*)a.s.tile_min;
        for (int tb = from / WT; tb < t1 && !a_done; tb += 32) {
          const bool tin = tb + lane < t1;
          const uint32_t tfl = tin ? __ldcg(&a.s.tile_flag[tb + lane]) : 0u;
          const T tmn = tin ? __ldcg(&tile_min_r[tb + lane]) : KeyTraits<T>::pad();
          unsigned fl = __ballot_sync(FULL, (tfl & 0x7fffffffu) != 0);
          while (fl && !a_done) {
            // Flagged tiles whose pending keys all take the cursor: not mixed, and
            // P and the cursor's key both qualify for the tile's minimum (<= every
            // pending key).  Pending keys do not increase, so these form a prefix
            // of the flagged tiles; their keys are not read.  A tile that is all
            // pending takes the cursor in 16-byte stores without its masks; of
            // the others the masks of 32/W tiles come in one load.
            const unsigned fast = __ballot_sync(
                FULL, ((fl >> lane) & 1u) && (tfl >> 31) == 0 && cur >= 0 && lt<INCL>(P, tmn) && lt<INCL>(cv, tmn));
            const unsigned slow = fl & ~fast;
            unsigned take = slow ? fl & ((slow & (0u - slow)) - 1u) : fl;
            fl &= ~take;
            unsigned whole = __ballot_sync(FULL, ((take >> lane) & 1u) && (tfl & 0x3fffffffu) == (uint32_t)WT &&
                                                     (tb + lane) * WT >= from && tile_full(tb + lane));
            take &= ~whole;
            while (whole) {
                const int t = tb + __ffs(whole) - 1;
                whole &= whole - 1;
#pragma unroll
                for (int j = 0; j < WT / 128; j++) put4(t * WT + 128 * j + 4 * lane, SEG ? seg_rel(cur, first_start) : cur);
            }
            while (take) {
                int tt[TPL], mine = -1;
#pragma unroll
                for (int h = 0; h < TPL; h++) {
                    tt[h] = take ? __ffs(take) - 1 : -1;
                    if (take) take &= take - 1;
                    if (lane / W == h) mine = tt[h];
                }
                const uint32_t mw2 = mine >= 0 ? __ldcg(&a.s.tile_mask[(size_t)(tb + mine) * MW + (lane % W)]) : 0u;
#pragma unroll
                for (int h = 0; h < TPL; h++) {
                    if (tt[h] < 0) break;
#pragma unroll
                    for (int w = 0; w < W; w++) {
                        const uint32_t mw = __shfl_sync(FULL, mw2, W * h + w);
                        const int pos = (tb + tt[h]) * WT + w * 32 + lane;
                        if (((mw >> lane) & 1u) && pos >= from && (!head || pos >= head))
                            put(pos, SEG ? seg_rel(cur, first_start) : cur);
                    }
                }
            }
            if (!fl) break;
            // The first other flagged tile: alone when it is mixed or all pending, else
            // with the tiles after it that are neither, up to a list of WT keys.
            const int fsrc = __ffs(fl) - 1;
            const int cnt = ((fl >> lane) & 1u) ? (int)(tfl & 0x3fffffffu) : 0;
            const bool alone = cnt == WT || (cnt && (tfl >> 31));
            int dummy;
            const int before = warp_excl_sum(min(cnt, WT), dummy);
            const unsigned stop = __ballot_sync(FULL, alone || before + cnt > WT);
            unsigned tk = stop ? fl & ((stop & (0u - stop)) - 1u) : fl;
            if ((stop >> fsrc) & 1u) {
                fl &= fl - 1;
                flagged_tile(tb + fsrc, (__shfl_sync(FULL, tfl, fsrc) >> 31) != 0, from, true);
                continue;
            }
            fl &= ~tk;
            int tot = 0;
            while (tk) {  // lists the keys: 4 * TPL tiles' masks in flight
                uint32_t mw[4];
                int mt[4];
#pragma unroll
                for (int p2 = 0; p2 < 4; p2++) {
                    mt[p2] = -1;
#pragma unroll
                    for (int h = 0; h < TPL; h++) {
                        if (lane / W == h && tk) mt[p2] = __ffs(tk) - 1;
                        tk &= tk - 1;
                    }
                    mw[p2] = mt[p2] >= 0 ? __ldcg(&a.s.tile_mask[(size_t)(tb + mt[p2]) * MW + (lane % W)]) : 0u;
                }
#pragma unroll
                for (int p2 = 0; p2 < 4; p2++) {
                    const int w0 = mt[p2] * WT + 32 * (lane % W);  // relative to tile tb
                    const int lim = max(from, head) - tb * WT;
                    if (w0 < lim) mw[p2] &= lim - w0 >= 32 ? 0u : (0xffffffffu << (lim - w0));
                    int n2;
                    int off = tot + warp_excl_sum(__popc(mw[p2]), n2);
                    for (uint32_t m = mw[p2]; m; m &= m - 1) sList[off++] = (int16_t)(w0 + __ffs(m) - 1);
                    tot += n2;
                }
            }
            __syncwarp();
            auto key_of = [&](const int j) {
                return j < tot ? key_at<T, MAPF, REV>(d_in, a.n, tb * WT + (int)sList[j]) : KeyTraits<T>::pad();
            };
            T qn = key_of(lane);
            for (int b0 = 0; b0 < tot && !a_done; b0 += 32) {
                const T q = qn;
                qn = key_of(b0 + 32 + lane);
                const bool in = b0 + lane < tot;
                deferred32(in, q, in ? tb * WT + (int)sList[b0 + lane] : 0);
            }
            __syncwarp();
          }
        }
    }

    // B. capped keys: the answer is in the range, below the stack's kept part.
    const int ncap = min(cap_total, kCapCap);
    for (int b0 = 0; b0 < ncap; b0 += 32) {
        const bool in = b0 + lane < ncap;
        const int pos = in ? sCapP[b0 + lane] : range_begin;
        const T q = in ? key_at<T, MAPF, REV>(d_in, a.n, pos) : KeyTraits<T>::pad();
        const int found = find_in_tiles<T, WT, INCL, MAPF, REV>(q, in, t0, pos / WT, true, d_in, a);
        if (in) {
            if (found < 0) atomicOr(err, ERR_INTERNAL);
            else if (!head || pos >= head) put(pos, SEG ? seg_rel(found, sCapS[b0 + lane]) : found);
        }
    }
    if (cap_total > kCapCap) {
        // B'. the capped list overflowed: every flagged key of the mixed tiles after it
        const int from = sCapP[kCapCap - 1] + 1;
        for (int tb = from / WT; tb < t1; tb += 32) {
            const uint32_t tfl = tb + lane < t1 ? __ldcg(&a.s.tile_flag[tb + lane]) : 0u;
            for (unsigned fl = __ballot_sync(FULL, (tfl >> 31) != 0); fl; fl &= fl - 1)
                flagged_tile(tb + __ffs(fl) - 1, true, from, false);
        }
    }
}

// MAPF: the key map (KMAP_*): keys stay as they landed in shared memory and pass
// through it as they are read -- float64 bit patterns in int64 slots compared through
// f64_order, or the order-reversing flip for previous-greater queries.
// OUTM (single arrays, no view head, except OUT_I32): OUT_I64 -- answers as
// int64, a.out_base + answer, into a.d_out64, for the int64-position path: a
// flagged key gets a.unanswered64 (phase 2 overwrites the ones it answers), and a
// tile whose keys are all deferred is not written at all (its flag word says
// so); the int64-position path answers what is left.  OUT_SPAN -- int32
// position - answer (position + 1 for none): the stock span, with the flip.
// REV (single arrays, no view head): the run sees the array
// reversed -- tile t holds elements n - 1 - (t * WT + e), its TMA rows counted
// from the end (n a multiple of 32) and read mirrored from shared
// memory -- and writes each answer mirrored back, n - 1 - answer (-1 for none)
// at element n - 1 - position: the next smaller key, in one run.

// Batches of 4-byte keys in 512-key tiles: less shared memory per warp, 20 warps per
// SM in configuration 0 (the segmented unit launches it so).
template <typename T, int IPT, bool SEG, bool EP>
constexpr bool kIsLean = SEG && !EP && IPT == 16 && sizeof(T) == 4;

// 16 warps per SM in every configuration: without the bound the 4-warp CTAs took
// 205 registers a thread and 8 warps fitted; with it, and a deferred list that
// lets four of their CTAs share an SM, 2^20 random-walk keys 34.7 -> 28.5 us.
template <typename T, int IPT, int WPC, bool INCL, bool SEG, bool EP, int MAPF = KMAP_NONE, int OUTM = OUT_I32,
          bool REV = false>
__global__ void __launch_bounds__(WPC * 32, WPC > 8 ? 1 : 16 / WPC)
apse_warp_kernel(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_out,
                 const RangeArgs a) {
    constexpr int KB = (int)sizeof(T);  // bytes per key
    constexpr bool LEAN = kIsLean<T, IPT, SEG, EP>;
    using L = WLayout<IPT, KB, LEAN>;
    constexpr int WT = L::WT;      // keys per warp tile
    constexpr int W = WT / 32;     // 32-key chunks (and answer TMA rows) per warp tile
    constexpr int RPT = W * KB / 4;  // key TMA rows (128 bytes) per warp tile
    constexpr int TPC = 32 / IPT;  // lanes per chunk
    constexpr int K = kStackCapOf<KB, LEAN>;
    constexpr int kStages = kStagesOf<KB, IPT>;
    constexpr int kDefCap = kDefCapOf<KB, IPT, LEAN>;
    constexpr int MW = kMaxTileKeys / 32;  // flag-mask words per tile in global
    static_assert(IPT == 8 || IPT == 16, "IPT must be 8 or 16");
    auto ks = [](int e) { return kswz<KB>(e); };  // swizzled index of key e in V / sSM
    static_assert((K & (K - 1)) == 0, "the stack ring needs a power-of-two size");
    static_assert(K % 32 == 0 && kUpKeep <= K && kUpKeep <= WT, "a whole-tile push copies the tile's last keys, 32 per step");
    constexpr unsigned FULL = 0xffffffffu;

    extern __shared__ unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    unsigned char* cta_sm = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* wsm = cta_sm + (size_t)warp * L::kBytes;
    // CTA words: [0] the CTA's first range, [1] warps of the CTA finished, [2] and [3]
    // see range_prefix
    int* sCta = (int*)(cta_sm + (size_t)WPC * L::kBytes);
    T* sV = (T*)(wsm + L::kV);
    int32_t* O = (int32_t*)(wsm + L::kO);
    T* sSM = (T*)(wsm + L::kSM);
    int16_t* sList = (int16_t*)(wsm + L::kList);
    T* sStkV = (T*)(wsm + L::kStkV);
    int32_t* sStkP = (int32_t*)(wsm + L::kStkP);
    int32_t* sDefP = (int32_t*)(wsm + L::kDefP);
    T* sDefV = (T*)(wsm + L::kDefV);
    int32_t* sCapP = (int32_t*)(wsm + L::kCapP);
    int32_t* sCapS = (int32_t*)(wsm + L::kCapS);
    T* sPad = (T*)(wsm + L::kPad);
    uint64_t* bar = (uint64_t*)(wsm + L::kBar);
    // 0, as a value the compiler does not know (grids are one-dimensional): see take_if_lt
    const int zero = (int)gridDim.y - 1;

    const T* d_in = (const T*)a.d_in;
    T* tile_min_w = (T*)a.s.tile_min;
    T* chunk_min_w = (T*)a.s.chunk_min;
    uint32_t* err = &a.s.ctr->err;
    // The view's virtual keys: only the segmented instantiations have them (a
    // batch off a 16-byte boundary; a single array off one runs as one implicit
    // segment with the whole-tile early paths, EP).
    const int head = SEG ? a.head : 0;
    // Segment offsets (positions in the array); with no offsets array, one segment.
    auto seg_off = [&](int i) -> int64_t {
        return a.offsets ? (int64_t)__ldg(&a.offsets[i]) : (i == 0 ? (int64_t)0 : (int64_t)(a.n - head));
    };
    auto seg_idx = [&](int pos) { return a.offsets ? seg_find(a.offsets, a.nseg, pos, err) : 0; };
    static_assert(OUTM == OUT_I32 || (!SEG && EP), "int64 and span answers: single arrays only");
    static_assert(!REV || (!SEG && EP && OUTM == OUT_I32), "reversed runs: single arrays");
    constexpr bool OUT64 = OUTM == OUT_I64;
    uint32_t epoch = 0;
    if (lane == 0) {
        for (int s = 0; s < kStages; s++) mbar_init(&bar[s], 1);
        for (int k = 0; k < 4; k++) sPad[k] = raw_pad<T, MAPF>();
        fence_mbarrier_init();
        fence_proxy_async_smem();
    }
    grid_dependency_wait();
    // One claim per CTA: its warps take WPC consecutive range ids, in the order
    // the CTAs start (so every range a warp may wait on belongs to a started CTA).
    if (threadIdx.x == 0) {
        sCta[0] = (int)atomicAdd(&a.s.ctr->range_counter, (unsigned)WPC);
        sCta[1] = sCta[2] = sCta[3] = 0;
    }
    if (lane == 0) epoch = ld_relaxed_u32(&a.s.ctr->epoch);
    __syncthreads();  // the CTA's claim is in shared memory
    const int r = sCta[0] + warp;
    epoch = __shfl_sync(FULL, epoch, 0);
    __syncwarp();

    if (r < a.num_ranges) {
        const int t0 = r * a.tiles_per_range;
        const int t1 = min(t0 + a.tiles_per_range, a.num_tiles);
        const int ntr = t1 - t0;
        auto tile_full = [&](int t) { return a.tma_rows > 0 && (t + 1) * RPT <= a.tma_rows && (t > 0 || head == 0); };
        // the first TMA row of tile t (reversed runs: counted from the end)
        auto tile_row = [&](int t) { return REV ? a.tma_rows - (t + 1) * RPT : t * RPT; };
        if (lane == 0) {
            for (int i = 0; i < kStages && i < ntr; i++)
                if (tile_full(t0 + i)) {
                    mbar_arrive_expect_tx(&bar[i], (uint32_t)(WT * KB));
                    tma_load_2d(sV + (size_t)i * WT, &map_in, 0, tile_row(t0 + i), &bar[i]);
                }
        }
        // Range state (warp-uniform): the stack ring [stk_lo, stk_hi) of strict
        // suffix minima, values increasing from bottom to top; whether entries were
        // ever dropped from its bottom; the range minimum so far; flagged-key counts.
        int stk_lo = 0, stk_hi = 0;
        bool dropped = false;
        bool has_rmin = false;
        T rmin = KeyTraits<T>::pad();
        int def_total = 0, cap_total = 0;
        // Segmented runs (warp-uniform): the segment at the cursor, its start and
        // the next segment start.
        int seg_cur = 0, cur_start = 0, next_b = INT_MAX;
        int first_start = 0, first_end = INT_MAX;  // the segment holding the range's first key
        if constexpr (SEG) {
            if (r == 0 && lane == 0 && a.offsets && (a.offsets[0] != 0 || a.offsets[a.nseg] != (int64_t)(a.n - head)))
                atomicOr(err, ERR_BAD_OFFSETS);
            // offsets are positions in the array; the view adds `head` virtual keys in
            // front (they fall in segment 0, and no answer of theirs is written)
            seg_cur = seg_idx(max(t0 * WT - head, 0));
            cur_start = (int)min(max(seg_off(seg_cur), (int64_t)0) + head, (int64_t)INT_MAX);
            next_b = (int)min(max(seg_off(seg_cur + 1), (int64_t)0) + head, (int64_t)INT_MAX);
            first_start = cur_start;
            first_end = next_b;
        }

        // ======================= phase 1: the range's tiles =======================
        for (int i = 0; i < ntr; i++) {
            const int t = t0 + i;
            const int slot = i % kStages;
            const uint32_t par = (uint32_t)((i / kStages) & 1);
            T* V = sV + (size_t)slot * WT;
            const bool full = tile_full(t);
            const int tile_base = t * WT;
            // Key e of the tile: the raw keys stay as they landed and go through the key map
            // as they are read; a reversed run sees them, and writes O, from the end
            // (reversing and mapping the tile in place cost 25-40 us at 2^25).
            auto at = [](int e) { return REV ? WT - 1 - e : e; };
            auto key = [&](int e) { return map_key<T, MAPF>(V[ks(at(e))]); };
            // the lane's 16-byte groups in element order, and the key at each place of them
            auto chunk = [&](int c) { return REV ? WT - (lane + 1) * IPT + c : lane * IPT + c; };
            auto in_chunk = [](int c) { return REV ? IPT - 1 - c : c; };
            // answers as they are written: reversed runs mirror them
            auto mirror = [&](int p) { return REV ? a.n - 1 - p : p; };
            const int valid_keys = min(WT, a.n - tile_base);

            if (full) {
                if (!mbar_wait_bounded(&bar[slot], par, a.spin_limit) && lane == 0) atomicOr(err, ERR_TMA_TIMEOUT);
            } else {
#pragma unroll
                for (int j = 0; j < IPT; j++) {
                    const int e = j * 32 + lane;
                    const int g = tile_base + e;
                    V[ks(at(e))] = g < a.n && (!head || g >= head) ? d_in[REV ? a.n - 1 - g : g] : raw_pad<T, MAPF>();
                }
                // A view head makes tile 0 plain while tile kStages streams into its
                // slot: the plain tile completes the slot barrier's phase by itself.
                // (Any other plain tile is the array's last: its slot is not reused.)
                if (head && lane == 0 && a.tma_rows > 0) mbar_arrive(&bar[slot]);
            }
            if (lane == 0) bulk_wait_read0();  // the previous tile's store has read O
            __syncwarp();
            // Every lane is done with V: the load of the tile kStages on goes there.
            auto load_ahead = [&]() {
                __syncwarp();
                if (lane == 0 && i + kStages < ntr && tile_full(t + kStages)) {
                    mbar_arrive_expect_tx(&bar[slot], (uint32_t)(WT * KB));
                    tma_load_2d(V, &map_in, 0, tile_row(t + kStages), &bar[slot]);
                }
            };

            // ---- 0. segmented runs: where segments start among the tile's keys ----------
            unsigned bword = 0;  // segment starts among this lane's keys (bit k: key k)
            int lane_s = 0;      // start of the segment holding this lane's first key
            // No segment starts inside the tile (most tiles): its answers are made relative
            // to the one start as they are found, with no pass over them before the store.
            bool one_seg = false;
            int rel = 0;  // that start (0 when answers are converted at the store)
            if constexpr (SEG) {
                const int tile_end = tile_base + WT;
                const int in_start = cur_start;
                if (next_b < tile_end) {
                    uint32_t* bm = (uint32_t*)sList;  // 512 bits; the X list is built later
                    if (lane < MW) bm[lane] = 0u;
                    __syncwarp();
                    for (int it = 0; it <= a.nseg / 32 + 1; it++) {  // ends once past off[nseg]
                        const int idx = seg_cur + 1 + lane;
                        const int64_t b = idx <= a.nseg ? seg_off(idx) + head : (int64_t)INT_MAX;
                        const bool in = b >= tile_base && b < tile_end;
                        if (in) atomicOr(&bm[(int)(b - tile_base) >> 5], 1u << ((int)(b - tile_base) & 31));
                        const int cnt = __popc(__ballot_sync(FULL, b < tile_end));
                        if (cnt) cur_start = (int)max((int64_t)0, __shfl_sync(FULL, b, cnt - 1));
                        seg_cur += cnt;
                        if (cnt < 32) {
                            next_b = (int)min((int64_t)INT_MAX, __shfl_sync(FULL, b, cnt));
                            break;
                        }
                    }
                    __syncwarp();
                    bword = (bm[(lane * IPT) >> 5] >> ((lane * IPT) & 31)) & (IPT == 32 ? 0xffffffffu : ((1u << IPT) - 1u));
                    int mx = bword ? tile_base + lane * IPT + 31 - __clz(bword) : -1;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int nb = __shfl_up_sync(FULL, mx, o);
                        if (lane >= o) mx = max(mx, nb);
                    }
                    const int before_b = __shfl_up_sync(FULL, mx, 1);
                    lane_s = max(in_start, lane > 0 ? before_b : -1);
                } else {
                    lane_s = in_start;
                    one_seg = in_start <= tile_base;  // (not so in the view's first tile)
                    rel = one_seg ? in_start : 0;
                }
            }
            // start of the segment holding key k of this lane
            auto seg_of = [&](int k) {
                const unsigned bb = bword & ((2u << k) - 1u);
                return bb ? tile_base + lane * IPT + 31 - __clz(bb) : lane_s;
            };

            // ---- 1. the lane's keys in registers ---------------------------------------
            T v[IPT];
            if constexpr (KB == 4) {
#pragma unroll
                for (int q4 = 0; q4 < IPT / 4; q4++) {
                    const uint4 rr = *reinterpret_cast<const uint4*>(&V[swz(chunk(4 * q4))]);
                    v[in_chunk(4 * q4 + 0)] = KeyTraits<T>::from_bits(rr.x);
                    v[in_chunk(4 * q4 + 1)] = KeyTraits<T>::from_bits(rr.y);
                    v[in_chunk(4 * q4 + 2)] = KeyTraits<T>::from_bits(rr.z);
                    v[in_chunk(4 * q4 + 3)] = KeyTraits<T>::from_bits(rr.w);
                }
            } else {  // two 8-byte keys per 16-byte chunk
#pragma unroll
                for (int q2 = 0; q2 < IPT / 2; q2++) {
                    const ulonglong2 rr = *reinterpret_cast<const ulonglong2*>(&V[ks(chunk(2 * q2))]);
                    v[in_chunk(2 * q2 + 0)] = KeyTraits<T>::from_bits((uint64_t)rr.x);
                    v[in_chunk(2 * q2 + 1)] = KeyTraits<T>::from_bits((uint64_t)rr.y);
                }
            }
            if constexpr (MAPF != KMAP_NONE) {
#pragma unroll
                for (int k = 0; k < IPT; k++) v[k] = map_key<T, MAPF>(v[k]);
            }
            const int lb = tile_base + lane * IPT;  // position of this lane's first key
            const int nvalid = min(max(a.n - lb, 0), IPT);
            // Flagged keys, deferred (dm) and capped (cm), keep -1 in O.  The first kDefCap
            // deferred and kCapCap capped keys of the range go to in-order lists in shared
            // memory for phase 2; every tile also leaves its flags in global memory for the
            // lists' overflow.
            auto flag_keys = [&](const unsigned dm, const unsigned cm) {
                {
                    const unsigned fm = dm | cm;
                    const int nd = __popc(dm), nc = __popc(cm);
                    const unsigned anyf = __ballot_sync(FULL, fm != 0);
                    int dtot = 0, ctot = 0;
                    if (anyf) {
                        const int doff = warp_excl_sum(nd, dtot);
                        const int coff = warp_excl_sum(nc, ctot);
                        {
                            int idx = def_total + doff;
                            unsigned m = dm;
                            while (m && idx < kDefCap) {
                                const int k = __ffs(m) - 1;
                                m &= m - 1;
                                sDefP[idx] = lb + k;
                                sDefV[idx] = key(lane * IPT + k);
                                idx++;
                            }
                        }
                        {
                            int idx = cap_total + coff;
                            unsigned m = cm;
                            while (m && idx < kCapCap) {
                                const int k = __ffs(m) - 1;
                                m &= m - 1;
                                if constexpr (SEG) sCapS[idx] = seg_of(k);
                                sCapP[idx++] = lb + k;
                            }
                        }
                        // mask word w covers keys [32w, 32w + 32): lanes TPC*w .. TPC*w + TPC - 1
                        uint32_t mw = 0;
    #pragma unroll
                        for (int j = 0; j < TPC; j++) {
                            const unsigned part = __shfl_sync(FULL, fm, (lane % W) * TPC + j);
                            mw |= part << (j * IPT);
                        }
                        if (lane < W) __stcg(&a.s.tile_mask[(size_t)t * MW + lane], mw);
                        def_total += dtot;
                        cap_total += ctot;
                    }
                    if (lane == 0) __stcg(&a.s.tile_flag[t], (uint32_t)(dtot + ctot) | (ctot ? 0x80000000u : 0u));
                }
            };
            // The whole tile leaves O, flagged keys as -1 (segmented runs: answers made
            // relative to their segment's start).
            auto store_tile = [&]() {
                if constexpr (OUT64) {  // int64 answers, 32 consecutive keys per store
                    __syncwarp();       // every lane's answers are in O
#pragma unroll
                    for (int j = 0; j < IPT; j++) {
                        const int e = j * 32 + lane;
                        if (e < valid_keys) {
                            const int o = O[swz(e)];
                            a.d_out64[tile_base + e] = o >= 0 ? (int64_t)o + a.out_base : a.unanswered64;
                        }
                    }
                    return;
                }
                if constexpr (OUTM == OUT_SPAN) {  // spans: position - answer
                    __syncwarp();                   // every lane's answers are in O
    #pragma unroll
                    for (int q4 = 0; q4 < IPT / 4; q4++) {
                        int4* po = reinterpret_cast<int4*>(&O[swz(lane * IPT + 4 * q4)]);
                        int4 o = *po;
                        const int p0 = tile_base + lane * IPT + 4 * q4;
                        o.x = p0 - o.x;
                        o.y = p0 + 1 - o.y;
                        o.z = p0 + 2 - o.z;
                        o.w = p0 + 3 - o.w;
                        *po = o;
                    }
                }
                if (SEG && !one_seg) {  // answers relative to their segment's start
                    __syncwarp();       // every lane's answers are in O
    #pragma unroll
                    for (int q4 = 0; q4 < IPT / 4; q4++) {
                        int4* po = reinterpret_cast<int4*>(&O[swz(lane * IPT + 4 * q4)]);
                        int4 o = *po;
                        o.x = seg_rel(o.x, seg_of(4 * q4 + 0));
                        o.y = seg_rel(o.y, seg_of(4 * q4 + 1));
                        o.z = seg_rel(o.z, seg_of(4 * q4 + 2));
                        o.w = seg_rel(o.w, seg_of(4 * q4 + 3));
                        *po = o;
                    }
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (full) {
                    if (lane == 0) {
                        tma_store_2d(&map_out, 0, REV ? a.tma_rows * 4 / KB - (t + 1) * W : t * W, O);
                        bulk_commit();
                    }
                } else {
    #pragma unroll
                    for (int j = 0; j < IPT; j++) {
                        const int e = j * 32 + lane;
                        if (e < valid_keys && (!head || tile_base + e >= head)) a.d_out[mirror(tile_base + e)] = O[swz(at(e))];
                    }
                }
            };

            // The four keys before the lane's first (lane 0: pads).
            T h[4];
            {
                const T* hp = lane > 0 ? &V[ks(REV ? WT - lane * IPT : lane * IPT - 4)] : sPad;
                if constexpr (KB == 4) {
                    const uint4 rr = *reinterpret_cast<const uint4*>(hp);
                    h[REV ? 3 : 0] = KeyTraits<T>::from_bits(rr.x);
                    h[REV ? 2 : 1] = KeyTraits<T>::from_bits(rr.y);
                    h[REV ? 1 : 2] = KeyTraits<T>::from_bits(rr.z);
                    h[REV ? 0 : 3] = KeyTraits<T>::from_bits(rr.w);
                } else {
                    const T* hq = lane > 0 ? &V[ks(REV ? WT - lane * IPT + 2 : lane * IPT - 2)] : sPad + 2;
                    const ulonglong2 r0 = *reinterpret_cast<const ulonglong2*>(hp);
                    const ulonglong2 r1 = *reinterpret_cast<const ulonglong2*>(hq);
                    h[REV ? 3 : 0] = KeyTraits<T>::from_bits((uint64_t)r0.x);
                    h[REV ? 2 : 1] = KeyTraits<T>::from_bits((uint64_t)r0.y);
                    h[REV ? 1 : 2] = KeyTraits<T>::from_bits((uint64_t)r1.x);
                    h[REV ? 0 : 3] = KeyTraits<T>::from_bits((uint64_t)r1.y);
                }
            }
            if constexpr (MAPF != KMAP_NONE) {
#pragma unroll
                for (int k = 0; k < 4; k++) h[k] = map_key<T, MAPF>(h[k]);
            }
            const T prev_last = h[3];

            // Monotone lanes: each key answers its neighbour (adj), or no key answers
            // any later one (none); across the lane boundary likewise (b_adj, b_none).
            // A few neighbour pairs first: on almost every tile of unordered keys some
            // lane is already neither increasing nor non-increasing there, and the
            // full check (15 compares a lane) and the whole-tile paths are skipped.
            bool adj = false, none = false, b_adj = false;
            unsigned mono = 0u;
            {
                bool qa = true, qn = true;
#pragma unroll
                for (int k = IPT / 4; k < IPT; k += IPT / 4) {
                    const bool l = lt<INCL>(v[k - 1], v[k]);
                    qa = qa && l;
                    qn = qn && !l;
                }
                if (__all_sync(FULL, qa || qn)) {
                    adj = true;
                    none = true;
#pragma unroll
                    for (int k = 1; k < IPT; k++) {
                        const bool l = lt<INCL>(v[k - 1], v[k]);
                        adj = adj && l;
                        none = none && !l;
                    }
                    mono = __ballot_sync(FULL, adj || none);
                    b_adj = lane == 0 || lt<INCL>(prev_last, v[0]);
                }
            }

            // ---- a whole tile below the range so far --------------------------------------
            // A tile that never increases (under the comparator, lane boundaries
            // included) and whose first key has no qualifying key earlier in the
            // range has no answer for any key inside the range: every key is deferred,
            // every stack entry (>= the range minimum >= the first key) is popped and
            // the tile's last key is its only strict suffix minimum.  (Single arrays,
            // also a single array behind a view head in the segmented kernel.)
            if (EP && mono == FULL && valid_keys == WT) {
                const T first = __shfl_sync(FULL, v[0], 0);
                const bool never = __all_sync(FULL, none && (lane == 0 || !b_adj));
                // No key of the tile answers another.  When the same entry of the stack's
                // top 32 is the topmost one to qualify for the tile's first and for its
                // last key, it answers every key between too (descending keys after a lower
                // one: 671 low keys in 2^25 descending ones sent a quarter of the ranges
                // through 16 rounds of stack queries a tile, 254 us against 51).
                unsigned same = 0u;  // the window entries that qualify for every key
                const int wlo = max(stk_lo, stk_hi - 32);
                T wtop = KeyTraits<T>::pad();
                const bool below = !has_rmin || !lt<INCL>(rmin, first);  // nothing in the range qualifies
                if (never && !below) {
                    const bool in = wlo + lane < stk_hi;
                    const T last = __shfl_sync(FULL, v[IPT - 1], 31);
                    wtop = in ? sStkV[(wlo + lane) & (K - 1)] : KeyTraits<T>::pad();
                    same = __ballot_sync(FULL, in && lt<INCL>(wtop, last));
                    if (same != __ballot_sync(FULL, in && lt<INCL>(wtop, first))) same = 0u;
                }
                if (same) {
                    const T tmin = __shfl_sync(FULL, v[IPT - 1], 31);
                    const int top = 31 - __clz(same);
                    const int tp = mirror(max(sStkP[(wlo + top) & (K - 1)] - (OUTM == OUT_I32 ? head : 0), -1));
#pragma unroll
                    for (int q4 = 0; q4 < IPT / 4; q4++)
                        *reinterpret_cast<int4*>(&O[swz(lane * IPT + 4 * q4)]) = make_int4(tp, tp, tp, tp);
                    if (((lane + 1) & (TPC - 1)) == 0) __stcg(&chunk_min_w[(size_t)t * W + lane / TPC], v[IPT - 1]);
                    if (lane == 0) {
                        __stcg(&a.s.tile_flag[t], 0u);
                        __stcg(&tile_min_w[t], tmin);
                    }
                    if constexpr (OUTM != OUT_I32 || REV) {
                        store_tile();
                    } else {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (full) {
                            if (lane == 0) {
                                tma_store_2d(&map_out, 0, t * W, O);
                                bulk_commit();
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < IPT; j++)
                                if (!head || tile_base + j * 32 + lane >= head) a.d_out[tile_base + j * 32 + lane] = tp;
                        }
                    }
                    __syncwarp();  // every lane has read the stack
                    // the entries below the tile's minimum stay (the top one may equal it
                    // under <=) and the tile's last key is pushed
                    const int kp = wlo + top + (__shfl_sync(FULL, wtop, top) < tmin ? 1 : 0);
                    if (lane == 31) {
                        sStkV[kp & (K - 1)] = v[IPT - 1];
                        sStkP[kp & (K - 1)] = tile_base + WT - 1;
                    }
                    stk_hi = kp + 1;
                    if (stk_hi - K > stk_lo) {
                        stk_lo = stk_hi - K;
                        dropped = true;
                    }
                    rmin = KeyTraits<T>::vmin(rmin, tmin);
                    load_ahead();
                    continue;
                }
                if (never && below) {
                    for (int e = lane; e < WT && def_total + e < kDefCap; e += 32) {
                        sDefP[def_total + e] = tile_base + e;
                        sDefV[def_total + e] = key(e);
                    }
                    // With nothing to store the loads set the pace, and the next one leaves
                    // here (2^28 keys in two pieces 636 -> 620 us); where the tile is stored
                    // too, loads this early made it slower (a run of 2^28: 372 -> 382 us).
                    if constexpr (OUT64) {
                        load_ahead();
                    } else {
                        const int4 m1 = make_int4(-1, -1, -1, -1);
#pragma unroll
                        for (int q4 = 0; q4 < IPT / 4; q4++) *reinterpret_cast<int4*>(&O[swz(lane * IPT + 4 * q4)]) = m1;
                    }
                    if (((lane + 1) & (TPC - 1)) == 0) __stcg(&chunk_min_w[(size_t)t * W + lane / TPC], v[IPT - 1]);
                    const T tmin = __shfl_sync(FULL, v[IPT - 1], 31);
                    if (lane < W) __stcg(&a.s.tile_mask[(size_t)t * MW + lane], 0xffffffffu);
                    if (lane == 0) {
                        __stcg(&a.s.tile_flag[t], (uint32_t)WT | (OUT64 ? TILE_NOT_STORED : 0u));
                        __stcg(&tile_min_w[t], tmin);
                    }
                    def_total += WT;
                    if constexpr (OUTM == OUT_SPAN || REV) {
                        store_tile();
                    } else if constexpr (!OUT64) {  // (int64 answers: the tile is left to the int64-position path)
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (full) {
                            if (lane == 0) {
                                tma_store_2d(&map_out, 0, t * W, O);
                                bulk_commit();
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < IPT; j++)
                                if (!head || tile_base + j * 32 + lane >= head) a.d_out[tile_base + j * 32 + lane] = -1;
                        }
                    }
                    if (lane == 31) {
                        sStkV[stk_lo & (K - 1)] = v[IPT - 1];
                        sStkP[stk_lo & (K - 1)] = tile_base + WT - 1;
                    }
                    stk_hi = stk_lo + 1;
                    rmin = tmin;
                    has_rmin = true;
                    if constexpr (OUT64) __syncwarp();
                    else load_ahead();
                    continue;
                }
            }

            // ---- a whole tile above the stack top ---------------------------------------------
            // A strictly increasing tile whose first key is above the stack's top entry
            // (the range's last key): every key answers its predecessor under either
            // comparator, every key is a strict suffix minimum, and the ring keeps the
            // tile's last kUpKeep keys.
            if (EP && mono == FULL && valid_keys == WT) {
                const T first = __shfl_sync(FULL, v[0], 0);
                bool up = __all_sync(FULL, adj && b_adj) && stk_hi > stk_lo && sStkV[(stk_hi - 1) & (K - 1)] < first;
                if constexpr (INCL) {
                    // adj means non-decreasing here: ties would not all be strict suffix
                    // minima, so check strict increase (only on such tiles)
                    if (up) {
                        bool inc = lane == 0 || prev_last < v[0];
#pragma unroll
                        for (int k = 1; k < IPT; k++) inc = inc && v[k - 1] < v[k];
                        up = __all_sync(FULL, inc);
                    }
                }
                if (up) {
                    // answers relative to the array (a view head's pads are never the
                    // stack top here: a pad does not lie below the tile's first key)
                    const int top_pos = sStkP[(stk_hi - 1) & (K - 1)] - head;
                    const int hb = lb - head;
                    auto up_ans = [&](int k) { return mirror(lane == 0 && k == 0 ? top_pos : hb + k - 1); };
#pragma unroll
                    for (int q4 = 0; q4 < IPT / 4; q4++)
                        *reinterpret_cast<int4*>(&O[swz(chunk(4 * q4))]) =
                            make_int4(up_ans(in_chunk(4 * q4)), up_ans(in_chunk(4 * q4 + 1)), up_ans(in_chunk(4 * q4 + 2)),
                                      up_ans(in_chunk(4 * q4 + 3)));
                    if ((lane & (TPC - 1)) == 0) __stcg(&chunk_min_w[(size_t)t * W + lane / TPC], v[0]);
                    if (lane == 0) {
                        __stcg(&a.s.tile_flag[t], 0u);
                        __stcg(&tile_min_w[t], first);
                    }
                    if constexpr (OUTM != OUT_I32 || REV) {
                        store_tile();
                    } else {
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (full) {
                            if (lane == 0) {
                                tma_store_2d(&map_out, 0, t * W, O);
                                bulk_commit();
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < IPT; j++)
                                if (!head || tile_base + j * 32 + lane >= head)
                                    a.d_out[tile_base + j * 32 + lane] = O[swz(j * 32 + lane)];
                        }
                    }
                    const int base_idx = stk_hi;  // entry of tile key e: base_idx + e
#pragma unroll
                    for (int h = 0; h < kUpKeep / 32; h++) {  // the tile's last keys, one per lane and step
                        const int e = WT - kUpKeep + h * 32 + lane;
                        sStkV[(base_idx + e) & (K - 1)] = key(e);
                        sStkP[(base_idx + e) & (K - 1)] = tile_base + e;
                    }
                    stk_hi = base_idx + WT;
                    stk_lo = stk_hi - kUpKeep;
                    dropped = true;  // the older entries are gone
                    rmin = KeyTraits<T>::vmin(rmin, first);
                    load_ahead();
                    continue;
                }
            }

            // Filled by the path below that handles the tile (steps 2-6, or a tile that never
            // increases) and used by steps 7-9.
            T tile_min_t = KeyTraits<T>::pad(), wv = KeyTraits<T>::pad();
            int win_lo = 0, dkeep = 0, ppre = 0, ptot = 0, fcnt = 0;
            unsigned fmask = 0;  // the lane's keys below every later key of the tile
            bool wvalid = false;
            // ---- a whole tile that never increases, above something earlier in the range -----
            // No key answers another, so every key's answer is the topmost qualifying entry
            // of the range stack (else it is capped or deferred), and as the keys do not
            // increase those entries only move down the stack: each lane searches the
            // stack for its first key, then walks down for the others.  The stack keeps
            // its entries below the tile's last key and takes that key.  Segmented
            // instantiations only (descending runs in batches of segments are made of
            // such tiles): in the single-array kernel the extra branch cost 5 us on
            // random keys at 2^25.
            const bool dtile =
                SEG && mono == FULL && valid_keys == WT && __all_sync(FULL, none && (lane == 0 || !b_adj));
            if (dtile) {
                unsigned dm = 0u, cm = 0u;
                const int dwin = max(stk_lo, stk_hi - 32);
                const int wcnt = stk_hi - dwin;
                const T dwv = dwin + lane < stk_hi ? sStkV[(dwin + lane) & (K - 1)] : KeyTraits<T>::pad();
                const T first = __shfl_sync(FULL, v[0], 0), last = __shfl_sync(FULL, v[IPT - 1], 31);
                const unsigned bl = __ballot_sync(FULL, lane < wcnt && lt<INCL>(dwv, last));
                const unsigned bf = __ballot_sync(FULL, lane < wcnt && lt<INCL>(dwv, first));
                int si;  // stack index of the current answer
                if (bl == bf && (bl || !(has_rmin && lt<INCL>(rmin, first)))) {
                    // the same window entry, or nothing in the range, answers every key (a tile
                    // inside one descending run; with the loop below per key a batch of such runs took
                    // 417 us instead of 314)
                    si = bl ? dwin + 31 - __clz(bl) : stk_lo - 1;
                    int rk = -1;
                    if (bl) rk = one_seg ? seg_rel(sStkP[si & (K - 1)], rel) : sStkP[si & (K - 1)];
                    else dm = IPT == 32 ? ~0u : (1u << IPT) - 1u;
#pragma unroll
                    for (int q4 = 0; q4 < IPT / 4; q4++)
                        *reinterpret_cast<int4*>(&O[swz(lane * IPT + 4 * q4)]) = make_int4(rk, rk, rk, rk);
                } else {
                int lo = -1;  // topmost qualifying window entry for the lane's first key
#pragma unroll
                for (int s2 = 32; s2 > 0; s2 >>= 1) {
                    const int cand = lo + s2;
                    const T wc = __shfl_sync(FULL, dwv, cand & 31);
                    if (cand < wcnt && lt<INCL>(wc, v[0])) lo = cand;
                }
                si = lo >= 0 ? dwin + lo : stk_lo - 1;
                if (lo < 0 && dwin > stk_lo) {  // below the window (values increase upwards)
                    int l2 = stk_lo, h2 = dwin;
                    while (l2 < h2) {
                        const int mid = (l2 + h2) >> 1;
                        if (lt<INCL>(sStkV[mid & (K - 1)], v[0])) l2 = mid + 1;
                        else h2 = mid;
                    }
                    si = l2 - 1;
                }
                // One rolled loop over the lane's keys, read back from the tile in shared
                // memory: with the loop unrolled over registers this path's code, beside
                // the general path's, overflowed the instruction cache when an SM's warps
                // ran both (a batch mixing descending runs with other keys: cache hit rate
                // 78 % -> 89 %, that batch 2.07 -> 1.93 ms; a batch of one long descending
                // run pays for the rolled loop instead, 0.88 -> 1.10 ms).
#pragma unroll 1
                for (int k = 0; k < IPT; k++) {
                    const T vk = key(lane * IPT + k);
                    if (k > 0)
                        while (si >= stk_lo && !lt<INCL>(sStkV[si & (K - 1)], vk)) si--;
                    int rk = -1;
                    if (si >= stk_lo) {
                        rk = one_seg ? seg_rel(sStkP[si & (K - 1)], rel) : sStkP[si & (K - 1)];
                    } else {
                        if (has_rmin && lt<INCL>(rmin, vk)) cm |= 1u << k;  // below the kept entries
                        else dm |= 1u << k;
                    }
                    O[swz(lane * IPT + k)] = rk;
                }
                }
                if constexpr (SEG) {  // deferred keys outside the range's first segment are final (-1)
                    if (lb + IPT > first_end) dm &= lb >= first_end ? 0u : ((1u << (first_end - lb)) - 1u);
                }
                if (cm && !dropped) atomicOr(err, ERR_INTERNAL);
                if (((lane + 1) & (TPC - 1)) == 0) __stcg(&chunk_min_w[(size_t)t * W + lane / TPC], v[IPT - 1]);
                tile_min_t = __shfl_sync(FULL, v[IPT - 1], 31);
                // the stack keeps its entries below the tile minimum (values >= it go; the
                // search's entry may equal it under <=) and takes the tile minimum
                int kp = __shfl_sync(FULL, si, 31);
                while (kp >= stk_lo && !(sStkV[kp & (K - 1)] < tile_min_t)) kp--;
                dkeep = kp + 1;
                flag_keys(dm, cm);
            } else {
            // ---- 2. in-thread answers: compare ladder ---------------------------------------
            // Key k of a lane against the lane's earlier keys, and its first keys also
            // against the 4 - k nearest ones before the lane, so that every key has seen
            // at least its four predecessors (10 compares a lane more; of 16 random keys
            // 2.1 instead of 3.4 are left for the cross-lane queries).  The compares are
            // what the ALU pipe does here; the selects go to the multiply-add pipe.
            unsigned umask = 0;  // keys without an in-thread answer: bit IPT - 1 - k for key k
            {
                int res[IPT];  // absolute answers, -1 = none in the thread
                const int lbo = lb - rel, mbo = mirror(lbo);
                if (mono == FULL) {  // monotone lanes need no ladder
                    res[0] = lane > 0 && b_adj ? mirror(lbo - 1) : -1;
#pragma unroll
                    for (int k = 1; k < IPT; k++) res[k] = adj ? mirror(lbo + k - 1) : -1;
                } else {
#pragma unroll
                    for (int k = 0; k < IPT; k++) {
                        int rk = REV ? mbo + 1 : -1 - lbo;  // relative to lbo
#pragma unroll
                        for (int j = k; j < 4; j++) take_if_lt<INCL>(rk, h[j], v[k], zero, j - 4);
#pragma unroll
                        for (int j = 0; j < k; j++) take_if_lt<INCL>(rk, v[j], v[k], zero, j);
                        res[k] = REV ? mbo - rk : rk + lbo;
                    }
                    if constexpr (INCL) {  // lane 0's pads qualify for keys of the pad's value
                        if (lane == 0)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (REV ? res[k] > mbo : res[k] < lbo) res[k] = -1;
                    }
                }
#pragma unroll
                for (int k = 0; k < IPT; k++) umask = __funnelshift_l((unsigned)res[k], umask, 1);
                if (nvalid < IPT) umask &= ~((1u << (IPT - nvalid)) - 1u);  // (the tail tile's pads)
                // in-thread answers; every other key holds -1 until resolved below
#pragma unroll
                for (int q4 = 0; q4 < IPT / 4; q4++)
                    *reinterpret_cast<int4*>(&O[swz(chunk(4 * q4))]) =
                        make_int4(res[in_chunk(4 * q4)], res[in_chunk(4 * q4 + 1)], res[in_chunk(4 * q4 + 2)],
                                  res[in_chunk(4 * q4 + 3)]);
            }
            // ---- 3. lane suffix minima, minima over lanes, the tile's strict suffix minima --
            T lmin, tab[5];
            {
                T sfx[IPT];  // suffix minima of the lane's keys (for the key search of X keys)
                sfx[IPT - 1] = v[IPT - 1];
#pragma unroll
                for (int k = IPT - 2; k >= 0; k--) sfx[k] = KeyTraits<T>::vmin(v[k], sfx[k + 1]);
                lmin = sfx[0];
                if constexpr (KB == 4) {
#pragma unroll
                    for (int q4 = 0; q4 < IPT / 4; q4++)
                        *reinterpret_cast<uint4*>(&sSM[swz(lane * IPT + 4 * q4)]) =
                            make_uint4(KeyTraits<T>::bits(sfx[4 * q4]), KeyTraits<T>::bits(sfx[4 * q4 + 1]),
                                       KeyTraits<T>::bits(sfx[4 * q4 + 2]), KeyTraits<T>::bits(sfx[4 * q4 + 3]));
                } else {
#pragma unroll
                    for (int q2 = 0; q2 < IPT / 2; q2++)
                        *reinterpret_cast<ulonglong2*>(&sSM[ks(lane * IPT + 2 * q2)]) =
                            make_ulonglong2((unsigned long long)KeyTraits<T>::bits(sfx[2 * q2]),
                                            (unsigned long long)KeyTraits<T>::bits(sfx[2 * q2 + 1]));
                }
                {
                    T cmn = lmin;
#pragma unroll
                    for (int o = 1; o < TPC; o <<= 1) cmn = KeyTraits<T>::vmin(cmn, __shfl_xor_sync(FULL, cmn, o));
                    if ((lane & (TPC - 1)) == 0) __stcg(&chunk_min_w[(size_t)t * W + lane / TPC], cmn);
                }
                // Side by side: suffix minima over lanes, and the lane table of the X
                // queries.  Slot s of the table stands for lane s - 1 (slot 0: a pad),
                // tab[k] = the minimum of slots (s - 2^k, s].
                T suf = lmin;
                tab[0] = __shfl_up_sync(FULL, lmin, 1);
                if (lane == 0) tab[0] = KeyTraits<T>::pad();
#pragma unroll
                for (int k = 0; k < 5; k++) {
                    const T na = __shfl_down_sync(FULL, suf, 1 << k);
                    if (lane + (1 << k) < 32) suf = KeyTraits<T>::vmin(suf, na);
                    if (k < 4) {
                        const T u = __shfl_up_sync(FULL, tab[k], 1 << k);
                        tab[k + 1] = lane >= (1 << k) ? KeyTraits<T>::vmin(tab[k], u) : tab[k];
                    }
                }
                tile_min_t = __shfl_sync(FULL, suf, 0);
                const T after_w = __shfl_down_sync(FULL, suf, 1);  // min of the lanes after (lane < 31)
                if (lane == 31 || lt<false>(lmin, after_w)) {      // else no key here beats every later key
#pragma unroll
                    for (int k = 0; k < IPT; k++)
                        if ((k == IPT - 1 || sfx[k] < sfx[k + 1]) && (lane == 31 || sfx[k] < after_w)) fmask |= 1u << k;
                }
            }
            // one prefix sum for both lists: keys to query, keys to push
            fcnt = __popc(fmask);
            ppre = warp_excl_sum(__popc(umask) | (fcnt << 16), ptot);
            const int qtot = ptot & 0xffff;
            win_lo = max(stk_lo, stk_hi - 32);  // the stack's top 32 entries, one per lane
            const int widx = win_lo + lane;
            wvalid = widx < stk_hi;
            wv = wvalid ? sStkV[widx & (K - 1)] : KeyTraits<T>::pad();
            const int wp = wvalid ? sStkP[widx & (K - 1)] : -1;

            // ---- 4. keys without an in-thread answer: an earlier lane of the tile (X) -------
            // Spread evenly over the lanes, up to NQ queries per lane and round: the lane by
            // binary lifting over the table, then the key by binary search of that lane's
            // suffix minima.  A query that ends on slot 0 or below has no answer in the tile;
            // those keys (in order) are left in the front of the list.
            int ns = 0, xtot = qtot;
            auto list_keys = [&](unsigned m, int off) {  // the keys of mask m, from list entry off on
                const int last_e = lane * IPT + IPT - 1;
                while (m) {
                    const int b = 31 - __clz(m);
                    m ^= 1u << b;
                    sList[off++] = (int16_t)(last_e - b);
                }
            };
            unsigned smask = 0u;  // keys known to have no answer in the tile
            int xoff = ppre & 0xffff;
            constexpr int NQ = kXQueries;
            T before = tab[4];  // the minimum of the lanes before
            {
                const T u = __shfl_up_sync(FULL, before, 16);
                if (lane >= 16) before = KeyTraits<T>::vmin(before, u);
            }
            // A lane's listed keys do not increase: when no earlier lane qualifies for its
            // first, none does for any.  No such key at all (ramps): nothing to query.
            const T q1 = key(lane * IPT + (IPT - 1 - (31 - __clz(umask | 1u))));
            if (!__any_sync(FULL, umask && lane > 0 && lt<INCL>(before, q1))) {
                smask = umask;
                xtot = xoff = 0;
            } else if (qtot > 32 * NQ) {
                // More than a round of keys: those no earlier lane qualifies for (most of
                // them, when keys fall) need no query.
#pragma unroll
                for (int k = 0; k < IPT; k++) smask = (smask << 1) | (lane > 0 && lt<INCL>(before, key(lane * IPT + k)) ? 0u : 1u);
                smask &= umask;
                xoff = warp_excl_sum(__popc(umask ^ smask), xtot);
            }
            list_keys(umask ^ smask, xoff);
            __syncwarp();  // in-thread answers, suffix minima and the list are in shared memory
            {
                for (int b0 = 0; b0 < xtot; b0 += 32 * NQ) {
                    int e[NQ], pl[NQ];
                    bool act[NQ];
                    T q[NQ];
#pragma unroll
                    for (int i2 = 0; i2 < NQ; i2++) {
                        act[i2] = b0 + 32 * i2 + lane < xtot;
                        e[i2] = act[i2] ? (int)sList[b0 + 32 * i2 + lane] : 0;
                    }
#pragma unroll
                    for (int i2 = 0; i2 < NQ; i2++) {
                        q[i2] = key(e[i2]);
                        pl[i2] = e[i2] / IPT;  // slot of the lane before the key's
                    }
                    // invariant: the answer's slot is <= pl and after each step pl - slot < 2^k;
                    // with no answer pl ends at 0 or below (a negative slot wraps to some
                    // lane's words: whatever they hold, pl stays negative)
#pragma unroll
                    for (int k = 4; k >= 0; k--) {
#pragma unroll
                        for (int i2 = 0; i2 < NQ; i2++) {
                            const T m = __shfl_sync(FULL, tab[k], pl[i2]);
                            if (!lt<INCL>(m, q[i2])) pl[i2] -= 1 << k;
                        }
                    }
                    // In lane pl - 1 the suffix minima qualify on a prefix [0, j] and key j is
                    // the answer; the lane's entries share one swizzle: word (lane*IPT | j) ^ x
                    int j[NQ], pb[NQ], px[NQ];
#pragma unroll
                    for (int i2 = 0; i2 < NQ; i2++) {
                        j[i2] = 0;
                        pb[i2] = max(pl[i2] - 1, 0) * IPT;
                        px[i2] = (pb[i2] >> 3) & (KB == 4 ? 0x1C : 0x0E);
                    }
#pragma unroll
                    for (int s2 = IPT / 2; s2 > 0; s2 >>= 1) {
#pragma unroll
                        for (int i2 = 0; i2 < NQ; i2++)
                            if (lt<INCL>(sSM[(pb[i2] | (j[i2] + s2)) ^ px[i2]], q[i2])) j[i2] += s2;
                    }
#pragma unroll
                    for (int i2 = 0; i2 < NQ; i2++) {
                        const bool out = act[i2] && pl[i2] <= 0;
                        if (act[i2] && !out) O[swz(at(e[i2]))] = mirror(tile_base - rel + pb[i2] + j[i2]);
                        const unsigned om = __ballot_sync(FULL, out);
                        if (out) sList[ns + __popc(om & ((1u << lane) - 1u))] = (int16_t)e[i2];
                        ns += __popc(om);
                    }
                    __syncwarp();
                }
            }
            if (xtot < qtot) {
                list_keys(smask, (ppre & 0xffff) - xoff);
                ns = qtot - xtot;
                __syncwarp();
            }

            // ---- 5. the rest: the range stack (S), else flagged: deferred or capped ---------
            // Stack entries are strict suffix minima: values increase from bottom to top
            // and the ones that qualify form a bottom part; the topmost of them answers.
            // With nothing ever dropped the bottom entry is the range minimum; a key that
            // the range minimum qualifies for but no kept entry is "capped" (phase 2 finds
            // its answer in the range), any other is "deferred" (nothing in the range
            // qualifies).  Flagged keys keep -1; they go to the lists of phase 2 and, for
            // the lists' overflow, as a mask per tile to global memory.
            int dtot = 0, ctot = 0;
            for (int b0 = 0; b0 < ns; b0 += 32) {
                const bool act = b0 + lane < ns;
                const int e = act ? (int)sList[b0 + lane] : 0;
                const T q = key(e);
                int ans = -1;
                if (__any_sync(FULL, act && has_rmin && lt<INCL>(rmin, q))) {
                    int lo = -1;  // the topmost qualifying entry of the window
#pragma unroll
                    for (int s2 = 32; s2 > 0; s2 >>= 1) {
                        const int cand = lo + s2;
                        const T wc = __shfl_sync(FULL, wv, cand & 31);
                        if (cand < stk_hi - win_lo && lt<INCL>(wc, q)) lo = cand;
                    }
                    ans = __shfl_sync(FULL, wp, lo & 31);
                    if (lo < 0) {
                        ans = -1;
                        if (act && win_lo > stk_lo) {  // below the window
                            int l2 = stk_lo, h2 = win_lo;
                            while (l2 < h2) {
                                const int mid = (l2 + h2) >> 1;
                                if (lt<INCL>(sStkV[mid & (K - 1)], q)) l2 = mid + 1;
                                else h2 = mid;
                            }
                            if (l2 > stk_lo) ans = sStkP[(l2 - 1) & (K - 1)];
                        }
                    }
                }
                if (act && ans >= 0) O[swz(at(e))] = SEG && one_seg ? seg_rel(ans, rel) : mirror(ans);
                const bool miss = act && ans < 0;
                if (__any_sync(FULL, miss)) {
                    const bool capd = miss && has_rmin && lt<INCL>(rmin, q);
                    bool defd = miss && !capd;
                    // Segmented: nothing in the range qualifies for a deferred key; if its
                    // segment starts inside the range, -1 is its final answer.
                    if constexpr (SEG) defd = defd && tile_base + e < first_end;
                    const unsigned db = __ballot_sync(FULL, defd), cb = __ballot_sync(FULL, capd);
                    if (db | cb) {
                        uint32_t* fm = (uint32_t*)sSM;  // the suffix minima are no longer needed
                        if (!(dtot | ctot)) {
                            if (lane < W) fm[lane] = 0u;
                            __syncwarp();
                        }
                        if (defd || capd) atomicOr(&fm[e >> 5], 1u << (e & 31));
                        const unsigned below = (1u << lane) - 1u;
                        const int di = def_total + dtot + __popc(db & below);
                        if (defd && di < kDefCap) {
                            sDefP[di] = tile_base + e;
                            sDefV[di] = q;
                        }
                        if (cb) {
                            if (!dropped) atomicOr(err, ERR_INTERNAL);
                            const int ci = cap_total + ctot + __popc(cb & below);
                            int sstart = 0;
                            if constexpr (SEG) {  // the start of the key's segment, from its lane
                                const unsigned bw = __shfl_sync(FULL, bword, e / IPT) & ((2u << (e % IPT)) - 1u);
                                sstart = __shfl_sync(FULL, lane_s, e / IPT);
                                if (bw) sstart = tile_base + e / IPT * IPT + 31 - __clz(bw);
                            }
                            if (capd && ci < kCapCap) {
                                sCapP[ci] = tile_base + e;
                                if constexpr (SEG) sCapS[ci] = sstart;
                            }
                        }
                        dtot += __popc(db);
                        ctot += __popc(cb);
                    }
                }
            }

            // ---- 6. flagged keys: the tile's mask and flag word -----------------------------
            if (dtot | ctot) {
                __syncwarp();
                if (lane < W) __stcg(&a.s.tile_mask[(size_t)t * MW + lane], ((const uint32_t*)sSM)[lane]);
                def_total += dtot;
                cap_total += ctot;
            }
            if (lane == 0) __stcg(&a.s.tile_flag[t], (uint32_t)(dtot + ctot) | (ctot ? 0x80000000u : 0u));
            }  // steps 2-6

            // ---- 7. output: the whole tile, flagged keys as -1 ----------------------------
            store_tile();

            // ---- 8. stack update: pop what the tile dominates, push its suffix minima ----
            if (dtile) {  // (the tile that never increases) push its minimum
                __syncwarp();  // every lane has read the stack
                if (lane == 31) {
                    sStkV[dkeep & (K - 1)] = v[IPT - 1];
                    sStkP[dkeep & (K - 1)] = tile_base + WT - 1;
                }
                stk_hi = dkeep + 1;
                if (stk_hi - K > stk_lo) {
                    stk_lo = stk_hi - K;
                    dropped = true;
                }
            } else {
                // Entries below the tile minimum survive: a bottom part of the stack.
                const unsigned below = __ballot_sync(FULL, wvalid && wv < tile_min_t);
                int keep;
                if (below == __ballot_sync(FULL, wvalid)) {
                    keep = stk_hi;  // the whole window survives, so does everything under it
                } else if (below || win_lo == stk_lo) {
                    keep = win_lo + __popc(below);
                } else {  // the boundary lies under the window (rare)
                    int lo = stk_lo, hi = win_lo;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (sStkV[mid & (K - 1)] < tile_min_t) lo = mid + 1;
                        else hi = mid;
                    }
                    keep = lo;
                }
                __syncwarp();  // every lane has read the old stack
                const int newtop = keep + (ptot >> 16);
                int idx = keep + (ppre >> 16);
                unsigned m = fmask;
                // Mostly the tile's last keys, all of them (a ramp): copied in key order, one
                // per lane, instead of up to IPT steps with every lane on its own keys.
                const int tot = ptot >> 16;
                if (tot >= 64) {
                    const int k0 = WT - tot - lane * IPT;  // the lane's first key to push
                    const unsigned all = (2u << (IPT - 1)) - 1u;
                    if (__all_sync(FULL, fmask == (k0 <= 0 ? all : k0 >= IPT ? 0u : all & (all << k0)))) {
                        for (int i2 = max(0, tot - K) + lane; i2 < tot; i2 += 32) {
                            sStkV[(keep + i2) & (K - 1)] = key(WT - tot + i2);
                            sStkP[(keep + i2) & (K - 1)] = tile_base + WT - tot + i2;
                        }
                        m = 0;
                    }
                }
                if (idx + fcnt <= newtop - K) m = 0;  // all of this lane's entries drop at once
                while (m) {
                    const int k = __ffs(m) - 1;
                    m &= m - 1;
                    if (idx >= newtop - K) {
                        sStkV[idx & (K - 1)] = key(lane * IPT + k);
                        sStkP[idx & (K - 1)] = lb + k;
                    }
                    idx++;
                }
                stk_hi = newtop;
                if (newtop - K > stk_lo) {
                    stk_lo = newtop - K;
                    dropped = true;
                }
            }

            // ---- 9. tile minimum, range minimum, next load ------------------------------
            if (lane == 0) __stcg(&tile_min_w[t], tile_min_t);
            rmin = has_rmin ? KeyTraits<T>::vmin(rmin, tile_min_t) : tile_min_t;
            has_rmin = true;
            load_ahead();
        }

        // ======================= publish the range, its prefix ======================
        {  // the top of the final stack, for later ranges' deferred keys
            const int tb = max(stk_lo, stk_hi - kTopEntries);
            const int tc = stk_hi - tb;
            T* top_key = (T*)a.s.top_key + (size_t)r * kTopEntries;
            int32_t* top_pos = a.s.top_pos + (size_t)r * kTopEntries;
            if (lane < tc) {
                __stcg(&top_key[lane], sStkV[(tb + lane) & (K - 1)]);
                __stcg(&top_pos[lane], sStkP[(tb + lane) & (K - 1)]);
            }
            if (lane == 0) __stcg(&a.s.top_cnt[r], (uint32_t)tc);
        }
        __syncwarp();  // every lane's words before lane 0's release in range_publish
        range_publish<T>(r, epoch, rmin, a);
        if (lane == 0) {  // (beside the wait for the other ranges)
            bulk_wait0();       // this range's tile stores have landed ...
            fence_proxy_async();  // ... before phase 2 overwrites flagged keys
        }
        T P, win;
        bool has_p;
        range_prefix<T>(r, epoch, a, sCta + 2, P, has_p, win);
        __syncwarp();  // lane 0's acquire and wait before every lane's reads and writes

        phase2<T, IPT, INCL, SEG, LEAN, MAPF, OUTM, REV>(a, wsm, r, t0, t1, def_total, cap_total, first_start, P, has_p, win);
    }

    // ---- run bookkeeping: the last warp resets the control block --------------------------
    // (the last warp of each CTA counts the CTA in; the last CTA resets)
    __syncwarp();
    int last = 0;
    if (lane == 0 && atomicAdd(&sCta[1], 1) == WPC - 1) {
        __threadfence();
        const uint32_t prev = atomicAdd(&a.s.ctr->done, 1u);
        last = prev == gridDim.x - 1;
        if (last) {
            a.s.ctr->range_counter = 0;
            a.s.ctr->done = 0;
            a.s.ctr->finished = 0;
            a.s.ctr->epoch = epoch >= EPOCH_LIMIT ? 1u : epoch + 1u;  // (the launch's end publishes these)
        }
    }
    last = __shfl_sync(FULL, last, 0);
    if (last && epoch >= EPOCH_LIMIT) {  // once per 2^30 runs: stale words could alias
        for (int i = lane; i < a.s.max_ranges; i += 32) a.s.range_state[i] = 0;
        for (int i = lane; i < a.s.max_ranges / 32; i += 32) a.s.group_min[i] = ~0ull;
    }
}

// ---------------------------------------------------------------------------
// Launch plumbing shared by the single-array and segmented translation units.
// ---------------------------------------------------------------------------
template <typename T, int IPT, int WPC, bool INCL, bool SEG, bool EP, int MAPF = KMAP_NONE, int OUTM = OUT_I32,
          bool REV = false>
inline cudaError_t launch_t(RangeArgs& a, const CUtensorMap& mi, const CUtensorMap& mo, cudaStream_t st,
                            int max_warps) {
    constexpr size_t smem = kernel_smem_bytes<IPT, WPC, (int)sizeof(T), kIsLean<T, IPT, SEG, EP>>();
    int tpr = (a.num_tiles + max_warps - 1) / max_warps;
    if (tpr < 1) tpr = 1;
    a.tiles_per_range = tpr;
    a.num_ranges = (a.num_tiles + tpr - 1) / tpr;
    const int ctas = (a.num_ranges + WPC - 1) / WPC;
    return launch_pdl(apse_warp_kernel<T, IPT, WPC, INCL, SEG, EP, MAPF, OUTM, REV>, ctas, WPC * 32, smem, st, mi, mo, a);
}

template <typename T, int IPT, int WPC, bool INCL, bool SEG, bool EP, int MAPF = KMAP_NONE, int OUTM = OUT_I32,
          bool REV = false>
inline cudaError_t prepare_t(int* ctas_per_sm) {
    constexpr size_t smem = kernel_smem_bytes<IPT, WPC, (int)sizeof(T), kIsLean<T, IPT, SEG, EP>>();
    auto k = apse_warp_kernel<T, IPT, WPC, INCL, SEG, EP, MAPF, OUTM, REV>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, WPC * 32, smem);
    if (e != cudaSuccess) return e;
    if (*ctas_per_sm == 0 || n < *ctas_per_sm) *ctas_per_sm = n;
    return cudaSuccess;
}

// Shared-memory attributes and occupancy of every kernel of one mode and
// configuration (the smallest CTAs-per-SM over the four key/comparison types).
template <bool SEG, bool EP>
inline cudaError_t prepare_mode(int cfg, int* per_sm) {
#define P_(IPT, WPC)                                                                   \
    {                                                                                  \
        cudaError_t rr[4] = {prepare_t<int32_t, IPT, WPC, false, SEG, EP>(per_sm),     \
                             prepare_t<int32_t, IPT, WPC, true, SEG, EP>(per_sm),      \
                             prepare_t<float, IPT, WPC, false, SEG, EP>(per_sm),       \
                             prepare_t<float, IPT, WPC, true, SEG, EP>(per_sm)};       \
        for (int q = 0; q < 4; q++)                                                    \
            if (rr[q] != cudaSuccess) return rr[q];                                    \
    }
    switch (cfg) {
    case 0:
        if constexpr (SEG && !EP) P_(16, kSegWarps) else P_(16, 16);
        break;
    case 1: P_(8, 8); break;
    case 2: P_(16, 8); break;
    case 3: P_(8, 16); break;
    case 4: P_(16, 4); break;
    case 5: P_(8, 4); break;
    default: return cudaErrorInvalidValue;
    }
#undef P_
    return cudaSuccess;
}

template <bool SEG, bool EP>
inline cudaError_t launch_mode(int dtype, int incl, int cfg, RangeArgs& a, const CUtensorMap& mi,
                               const CUtensorMap& mo, cudaStream_t st, int max_warps) {
#define L_(IPT, WPC)                                                                        \
    if (dtype == 0)                                                                         \
        return incl ? launch_t<int32_t, IPT, WPC, true, SEG, EP>(a, mi, mo, st, max_warps)  \
                    : launch_t<int32_t, IPT, WPC, false, SEG, EP>(a, mi, mo, st, max_warps); \
    else                                                                                    \
        return incl ? launch_t<float, IPT, WPC, true, SEG, EP>(a, mi, mo, st, max_warps)    \
                    : launch_t<float, IPT, WPC, false, SEG, EP>(a, mi, mo, st, max_warps);
    switch (cfg) {
    case 0:
        if constexpr (SEG && !EP) {
            L_(16, kSegWarps)
        } else {
            L_(16, 16)
        }
    case 1: L_(8, 8);
    case 2: L_(16, 8);
    case 3: L_(8, 16);
    case 4: L_(16, 4);
    case 5: L_(8, 4);
    }
#undef L_
    return cudaErrorInvalidValue;
}

}  // namespace apsep
