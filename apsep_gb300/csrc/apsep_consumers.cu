// apsep_consumers.cu -- the classic callers of APSE, built on the engine.
//
// Previous greater, next smaller, stock span, largest rectangle in a
// histogram and Cartesian-tree parents are all nearest-smaller queries in
// disguise (the reference names them as the consumers of its output,
// README.md:3, src/bench_spt_le.cu:1-3):
//   previous greater  = APSE of the order-reversed keys (int: ~x, float: -x)
//   next smaller      = APSE of the reversed array, answers mirrored back
//   stock span        = i - previous strictly greater
//   largest rectangle = max over i of h[i] * (next smaller - previous smaller - 1)
//   Cartesian parent  = of previous smaller-or-equal and next smaller, the one
//                       with the larger key (ties: the next one)
// With 4-byte keys on a 16-byte boundary, and 8-byte ones in arrays of long tiles,
// the engine does the flips and reversals itself (apsep_mapped.cu,
// apsep_wide_mapped.cu): previous greater and the stock span are
// one run each with the keys flipped as they load (and position - answer as
// the answers leave), next smaller one run over the reversed array with its
// answers mirrored as they leave (the last n % 32 keys apart: a pass over the answers
// completes them from those), and the histogram and
// Cartesian tree take that run for their next-smaller half.  Otherwise each is
// a few memory-bound passes (flip / reverse / mirror / epilogue, grid-stride,
// coalesced) around one or two engine runs.  All run on the caller's plan and
// stream with a caller-provided workspace: no allocation, no synchronisation,
// graph-capturable like apsep_run.
#include <stdint.h>

#include <type_traits>

#include "apsep.h"
#include "apsep_device.cuh"
#include "apsep_internal.h"

namespace {

constexpr int kThreads = 256;

int grid_for(int64_t n) {
    const int64_t b = (n + kThreads * 4 - 1) / (kThreads * 4);  // ~4 elements per thread
    return (int)(b < 1 ? 1 : b > 152 * 16 ? 152 * 16 : b);
}

size_t align16(size_t x) { return (x + 15) / 16 * 16; }

// Order-reversing map: a < b  <=>  flip(a) > flip(b), exactly (int: ~x = -x-1;
// float: -x, the two zeros stay equal).
__device__ __forceinline__ int32_t flip(int32_t x) { return ~x; }
__device__ __forceinline__ float flip(float x) { return -x; }
__device__ __forceinline__ int64_t flip(int64_t x) { return ~x; }
__device__ __forceinline__ double flip(double x) { return -x; }

int key_bytes(int dtype) { return dtype == APSEP_INT64 || dtype == APSEP_FLOAT64 ? 8 : 4; }

// Calls f(T*) with a null pointer of the plan's key type.
template <typename F>
void for_key_type(int dtype, F&& f) {
    switch (dtype) {
    case APSEP_INT32: f((int32_t*)nullptr); break;
    case APSEP_FLOAT32: f((float*)nullptr); break;
    case APSEP_INT64: f((int64_t*)nullptr); break;
    default: f((double*)nullptr); break;
    }
}

// Workspace: the keys (n of the plan's type), then two answer arrays.
struct Work {
    void* keys;
    int32_t* a;
    int32_t* b;
};
Work carve(void* d_work, int64_t n, int dtype) {
    char* w = (char*)d_work;
    const size_t kb = align16((size_t)n * key_bytes(dtype)), ab = align16((size_t)n * 4);
    return {w, (int32_t*)(w + kb), (int32_t*)(w + kb + ab)};
}

// Runs use(i, load(i)) for every i < n over the grid, kBatch loads of a thread in
// flight before the first use: these passes wait for memory, not for instructions
// (2^24 + 5 int32 keys, one load at a time against four: next smaller 94 | 86 us,
// Cartesian parents 202 | 182, of which two thirds are the engine's runs).
constexpr int kBatch = 4;
template <typename L, typename U>
__device__ __forceinline__ void for_batches(int64_t n, L load, U use) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kBatch * stride) {
        decltype(load(i0)) v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++)
            if (i0 + u * stride < n) v[u] = load(i0 + u * stride);
#pragma unroll
        for (int u = 0; u < kBatch; u++)
            if (i0 + u * stride < n) use(i0 + u * stride, v[u]);
    }
}

template <typename T>
__global__ void flip_keys(const T* __restrict__ in, T* __restrict__ out, int64_t n) {
    apsep::grid_dependency_wait();
    for_batches(n, [&](int64_t i) { return in[i]; }, [&](int64_t i, T v) { out[i] = flip(v); });
}

template <typename T>
__global__ void reverse_keys(const T* __restrict__ in, T* __restrict__ out, int64_t n) {
    apsep::grid_dependency_wait();
    for_batches(n, [&](int64_t i) { return in[n - 1 - i]; }, [&](int64_t i, T v) { out[i] = v; });
}

// The next-smaller answer from its mirror image, a previous-smaller answer of the
// reversed array (-1: none).
__device__ __forceinline__ int64_t next_from_reversed(int32_t a, int64_t n) { return a >= 0 ? n - 1 - a : -1; }
// A key as these passes compare it: float64 keys by the order-preserving map of their
// bits (each thread's minimum over a tail of 25 keys, compared as doubles, took next
// smaller of 5M float64 keys from 56 to 83 us).
template <typename T>
__device__ __forceinline__ T ordered(T x) {
    return x;
}
__device__ __forceinline__ int64_t ordered(double x) { return apsep::f64_order(__double_as_longlong(x)); }
template <typename T>
using Ordered = std::conditional_t<std::is_same_v<T, double>, int64_t, T>;
// The keys after the last multiple of 32 (the engine's reversed run takes whole
// 32-key rows): at most 31 of them, in shared memory, with their minimum.
template <typename K>
struct Tail {
    const K* v;
    K least;
    int count;
    int64_t base;  // position of the first (n when there is none)
};
// Called by every thread of the block; v: 32 keys of its shared memory.
template <typename T>
__device__ __forceinline__ Tail<Ordered<T>> load_tail(const T* __restrict__ a, int64_t n, int64_t base,
                                                      Ordered<T>* v) {
    const int count = (int)(n - base);
    if ((int)threadIdx.x < count) v[threadIdx.x] = ordered(a[base + threadIdx.x]);
    __syncthreads();
    Ordered<T> least = count > 0 ? v[0] : Ordered<T>(0);
    for (int j = 1; j < count; j++) least = v[j] < least ? v[j] : least;
    return {v, least, count, base};
}
// The first tail key at or after position i that is smaller (or equal) than q, or -1.
template <bool LE, typename K>
__device__ __forceinline__ int64_t next_in_tail(const Tail<K>& t, K q, int64_t i) {
    if (t.count == 0 || !(LE ? t.least <= q : t.least < q)) return -1;
    for (int j = i > t.base ? (int)(i - t.base) : 0; j < t.count; j++)
        if (LE ? t.v[j] <= q : t.v[j] < q) return t.base + j;
    return -1;
}
// What next-smaller answer of key i to load (next_word) and its meaning (next_of): R
// holds the answers themselves over the keys before the tail (direct, a reversed run of
// the engine), or the reversed array's previous-smaller answers (no tail).
template <typename K>
__device__ __forceinline__ int32_t next_word(const int32_t* __restrict__ R, bool direct, const Tail<K>& t, int64_t n,
                                             int64_t i) {
    return !direct ? R[n - 1 - i] : i < t.base ? R[i] : -1;
}
template <typename T>
__device__ __forceinline__ int64_t next_of(const T* __restrict__ a, int32_t word, bool direct,
                                           const Tail<Ordered<T>>& t, int64_t n, int64_t i) {
    if (!direct) return next_from_reversed(word, n);
    return word >= 0 || t.count == 0 ? word : next_in_tail<false>(t, ordered(a[i]), i + 1);
}

// Completes next-smaller answers of a reversed run over the keys before the tail:
// its unanswered keys and the tail's own.
template <typename T, bool LE>
__global__ void next_with_tail(const T* __restrict__ a, int32_t* __restrict__ out, int64_t n, int64_t base) {
    __shared__ Ordered<T> tail_keys[32];
    apsep::grid_dependency_wait();
    const Tail<Ordered<T>> t = load_tail(a, n, base, tail_keys);
    for_batches(
        n, [&](int64_t i) { return i < base ? out[i] : -1; },
        [&](int64_t i, int32_t r) {
            if (r >= 0) return;
            const int64_t o = next_in_tail<LE>(t, ordered(a[i]), i + 1);
            if (o >= 0 || i >= base) out[i] = (int32_t)o;  // (a key without one reads -1 already)
        });
}

__global__ void mirror_answers(const int32_t* __restrict__ ar, int32_t* __restrict__ out, int64_t n) {
    apsep::grid_dependency_wait();
    for_batches(
        n, [&](int64_t i) { return ar[n - 1 - i]; },
        [&](int64_t i, int32_t r) { out[i] = (int32_t)next_from_reversed(r, n); });
}

__global__ void span_from_previous(int32_t* __restrict__ a, int64_t n) {
    apsep::grid_dependency_wait();
    for_batches(n, [&](int64_t i) { return a[i]; }, [&](int64_t i, int32_t p) { a[i] = (int32_t)(i - p); });
}

// max over i of h[i] * (R - L - 1): L previous strictly smaller (-1: none), R
// next strictly smaller (n: none).  Only positive areas compete (heights are
// non-negative by contract; a negative height contributes nothing).
__global__ void rect_area(const int32_t* __restrict__ h, const int32_t* __restrict__ L,
                          const int32_t* __restrict__ ar, bool direct, int64_t base, int64_t n,
                          unsigned long long* __restrict__ best) {
    __shared__ long long warp_best[kThreads / 32];
    __shared__ int32_t tail_keys[32];
    apsep::grid_dependency_wait();
    const Tail<int32_t> t = load_tail(h, n, base, tail_keys);
    long long m = 0;
    for_batches(
        n, [&](int64_t i) { return int3{h[i], L[i], next_word(ar, direct, t, n, i)}; },
        [&](int64_t i, int3 v) {
            const int64_t r = next_of(h, v.z, direct, t, n, i);
            const int64_t w = (r < 0 ? n : r) - (int64_t)v.y - 1;
            const long long area = (long long)v.x * w;
            m = area > m ? area : m;
        });
    for (int o = 16; o > 0; o >>= 1) {
        const long long u = __shfl_xor_sync(0xffffffffu, m, o);
        m = u > m ? u : m;
    }
    if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long b = 0;
        for (int w = 0; w < kThreads / 32; w++) b = warp_best[w] > b ? warp_best[w] : b;
        if (b > 0) atomicMax(best, (unsigned long long)b);
    }
}

// Min-rooted Cartesian tree, ties as the stack construction makes them (a
// later equal key is the right child of an earlier one): L previous
// smaller-or-equal, R next strictly smaller; the parent is the one with the
// larger key, R on a tie; -1 for the root.
template <typename T>
__global__ void cartesian_parent(const T* __restrict__ a, const int32_t* __restrict__ L,
                                 const int32_t* __restrict__ ar, bool direct, int64_t base,
                                 int32_t* __restrict__ out, int64_t n) {
    __shared__ Ordered<T> tail_keys[32];
    apsep::grid_dependency_wait();
    const Tail<Ordered<T>> t = load_tail(a, n, base, tail_keys);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kBatch * stride) {
        // kBatch keys of a thread side by side: the answers' reads, then their keys'
        int32_t l[kBatch], r[kBatch];
        Ordered<T> kl[kBatch], kr[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int64_t i = i0 + u * stride;
            l[u] = i < n ? L[i] : -1;
            r[u] = i < n ? next_word(ar, direct, t, n, i) : -1;
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int64_t i = i0 + u * stride;
            if (i < n) r[u] = (int32_t)next_of(a, r[u], direct, t, n, i);
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            kl[u] = ordered(a[l[u] < 0 ? 0 : l[u]]);
            kr[u] = ordered(a[r[u] < 0 ? 0 : r[u]]);
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int64_t i = i0 + u * stride;
            if (i < n) out[i] = r[u] < 0 ? l[u] : l[u] < 0 || kr[u] >= kl[u] ? r[u] : l[u];
        }
    }
}

bool overlaps(const void* a, size_t an, const void* b, size_t bn) {
    const uintptr_t a0 = (uintptr_t)a, b0 = (uintptr_t)b;
    return a0 < b0 + bn && b0 < a0 + an;
}

// The reversed run of the engine over the keys before the last n % 32, when it has
// that form for the call (whole rows of 32 keys; *base: where they end), else
// APSEP_ENOTSUP.
apsep_status run_reversed(apsep_plan* plan, int dtype, const void* d_in, int32_t* d_out, int64_t n, apsep_cmp cmp,
                          void* stream, int64_t* base) {
    *base = n / 32 * 32;
    if (*base == 0 || overlaps(d_in, (size_t)n * key_bytes(dtype), d_out, (size_t)n * 4)) return APSEP_ENOTSUP;
    return plan_run_reversed(plan, d_in, d_out, *base, cmp, stream);
}

// Common argument checks; fills the plan's key type.
apsep_status check_args(apsep_plan* plan, const void* d_in, const void* d_out, size_t out_bytes, int64_t n,
                        void* d_work, int* dtype) {
    if (!plan || n < 0) return APSEP_EINVAL;
    apsep_plan_info info;
    const apsep_status s = apsep_plan_get_info(plan, &info);
    if (s != APSEP_OK) return s;
    *dtype = info.dtype;
    if (n == 0) return APSEP_OK;
    if (n > info.capacity || !d_in || !d_out || !d_work) return APSEP_EINVAL;
    const size_t kb = (size_t)n * key_bytes(info.dtype);
    if ((uintptr_t)d_work % 16 != 0 || (uintptr_t)d_in % key_bytes(info.dtype) != 0) return APSEP_EINVAL;
    const size_t wb = (size_t)apsep_consumer_workspace_bytes(n);
    if (overlaps(d_work, wb, d_in, kb) || overlaps(d_work, wb, d_out, out_bytes)) return APSEP_EINVAL;
    return APSEP_OK;
}

// Launches a grid-stride kernel over n elements.
template <typename K, typename... A>
apsep_status launched(K kernel, int64_t n, cudaStream_t st, const A&... args) {
    return apsep::launch_pdl(kernel, grid_for(n), kThreads, 0, st, args...) == cudaSuccess ? APSEP_OK : APSEP_ECUDA;
}

}  // namespace

extern "C" {

int64_t apsep_consumer_workspace_bytes(int64_t n) {
    if (n < 0) return 0;
    return (int64_t)(align16((size_t)n * 8) + 2 * align16((size_t)n * 4));  // any key type
}

apsep_status apsep_run_prev_greater(apsep_plan* plan, const void* d_in, int32_t* d_out, int64_t n, apsep_cmp cmp,
                                    void* d_work, void* stream) {
    int dtype = 0;
    apsep_status s = check_args(plan, d_in, d_out, (size_t)n * 4, n, d_work, &dtype);
    if (s != APSEP_OK || n == 0) return s;
    // one engine run that flips the keys as it loads them, when it has that form for
    // the call, else a flip pass into the workspace and a plain run
    if ((s = plan_run_flipped(plan, d_in, d_out, n, cmp, 0, stream)) != APSEP_ENOTSUP) return s;
    const cudaStream_t st = (cudaStream_t)stream;
    for_key_type(dtype, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        s = launched(flip_keys<T>, n, st, (const T*)d_in, (T*)d_work, n);
    });
    if (s != APSEP_OK) return s;
    return apsep_run_cmp(plan, d_work, d_out, n, cmp, stream);
}

apsep_status apsep_run_next_smaller(apsep_plan* plan, const void* d_in, int32_t* d_out, int64_t n, apsep_cmp cmp,
                                    void* d_work, void* stream) {
    int dtype = 0;
    apsep_status s = check_args(plan, d_in, d_out, (size_t)n * 4, n, d_work, &dtype);
    if (s != APSEP_OK || n == 0) return s;
    // one engine run over the reversed array, answers mirrored as they leave,
    // when it has that form for the call; else reverse, run, mirror
    const cudaStream_t st = (cudaStream_t)stream;
    int64_t base = n;
    if ((s = run_reversed(plan, dtype, d_in, d_out, n, cmp, stream, &base)) != APSEP_ENOTSUP) {
        if (s != APSEP_OK || base == n) return s;
        const bool le = cmp == APSEP_LE;
        for_key_type(dtype, [&](auto tag) {
            using T = std::remove_pointer_t<decltype(tag)>;
            s = launched(le ? next_with_tail<T, true> : next_with_tail<T, false>, n, st, (const T*)d_in, d_out, n, base);
        });
        return s;
    }
    const Work w = carve(d_work, n, dtype);
    for_key_type(dtype, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        s = launched(reverse_keys<T>, n, st, (const T*)d_in, (T*)w.keys, n);
    });
    if (s != APSEP_OK) return s;
    if ((s = apsep_run_cmp(plan, w.keys, w.a, n, cmp, stream)) != APSEP_OK) return s;
    s = launched(mirror_answers, n, st, w.a, d_out, n);
    return s;
}

apsep_status apsep_stock_span(apsep_plan* plan, const void* d_in, int32_t* d_out, int64_t n, void* d_work,
                              void* stream) {
    int dtype = 0;
    apsep_status s = check_args(plan, d_in, d_out, (size_t)n * 4, n, d_work, &dtype);
    if (s != APSEP_OK || n == 0) return s;
    // one engine run that flips the keys as it loads them and writes
    // position - answer, when it has that form for the call
    if ((s = plan_run_flipped(plan, d_in, d_out, n, APSEP_LT, 1, stream)) != APSEP_ENOTSUP) return s;
    s = apsep_run_prev_greater(plan, d_in, d_out, n, APSEP_LT, d_work, stream);
    if (s != APSEP_OK || n == 0) return s;
    s = launched(span_from_previous, n, (cudaStream_t)stream, d_out, n);
    return s;
}

apsep_status apsep_largest_rectangle(apsep_plan* plan, const int32_t* d_heights, int64_t n, int64_t* d_area,
                                     void* d_work, void* stream) {
    int dtype = 0;
    apsep_status s = check_args(plan, d_heights, d_area, 8, n, d_work, &dtype);
    if (s != APSEP_OK) return s;
    if (dtype != APSEP_INT32) return APSEP_ENOTSUP;
    if (!d_area || (uintptr_t)d_area % 8 != 0) return APSEP_EINVAL;
    const cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(d_area, 0, 8, st) != cudaSuccess) return APSEP_ECUDA;
    if (n == 0) return APSEP_OK;
    const Work w = carve(d_work, n, dtype);
    if ((s = apsep_run_cmp(plan, d_heights, w.b, n, APSEP_LT, stream)) != APSEP_OK) return s;
    // next smaller: one reversed run when the engine has that form, else
    // reverse the heights and run (the answers then come mirrored)
    bool direct = true;
    int64_t base = n;  // where the tail begins (none after a run over the whole reversed copy)
    if ((s = run_reversed(plan, dtype, d_heights, w.a, n, APSEP_LT, stream, &base)) == APSEP_ENOTSUP) {
        direct = false;
        base = n;
        s = launched(reverse_keys<int32_t>, n, st, d_heights, (int32_t*)w.keys, n);
        if (s != APSEP_OK) return s;
        s = apsep_run_cmp(plan, w.keys, w.a, n, APSEP_LT, stream);
    }
    if (s != APSEP_OK) return s;
    s = launched(rect_area, n, st, d_heights, w.b, w.a, direct, base, n, (unsigned long long*)d_area);
    return s;
}

apsep_status apsep_cartesian_parents(apsep_plan* plan, const void* d_in, int32_t* d_out, int64_t n, void* d_work,
                                     void* stream) {
    int dtype = 0;
    apsep_status s = check_args(plan, d_in, d_out, (size_t)n * 4, n, d_work, &dtype);
    if (s != APSEP_OK || n == 0) return s;
    const cudaStream_t st = (cudaStream_t)stream;
    const Work w = carve(d_work, n, dtype);
    if ((s = apsep_run_cmp(plan, d_in, w.b, n, APSEP_LE, stream)) != APSEP_OK) return s;
    bool direct = true;  // next smaller straight from a reversed run, else mirrored
    int64_t base = n;
    if ((s = run_reversed(plan, dtype, d_in, w.a, n, APSEP_LT, stream, &base)) == APSEP_ENOTSUP) {
        direct = false;
        base = n;
        for_key_type(dtype, [&](auto tag) {
            using T = std::remove_pointer_t<decltype(tag)>;
            s = launched(reverse_keys<T>, n, st, (const T*)d_in, (T*)w.keys, n);
        });
        if (s != APSEP_OK) return s;
        s = apsep_run_cmp(plan, w.keys, w.a, n, APSEP_LT, stream);
    }
    if (s != APSEP_OK) return s;
    for_key_type(dtype, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        s = launched(cartesian_parent<T>, n, st, (const T*)d_in, w.b, w.a, direct, base, d_out, n);
    });
    return s;
}

}  // extern "C"
