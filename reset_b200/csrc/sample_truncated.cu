// Top-k / top-p sampling of one id per row in one launch: one thread-block cluster of eight CTAs per row.
//
// The row is read from memory once; each CTA keeps an eighth of it in shared memory and the eight exchange
// histograms, totals and picks through distributed shared memory with cluster barriers. Phases:
//   1. load, row maximum, and a lower bound of the k-th largest value;
//   2. per truncation (top-k by count, then top-p by mass) a radix descent over the order-preserving keys,
//      11 + 11 + 10 bits: histogram of the keys that share the prefix found so far, each CTA sums 256 of the
//      2048 bins over the eight histograms, and the CTA whose bins cross the goal announces the bin. After
//      the last level the prefix is the key of the last token kept; equal keys are all kept;
//   3. arg-max of logit + Gumbel noise among the keys at or above the threshold.
// Mass is exp(x - row max) scaled by 2^32 and truncated to an integer, so no result depends on the order of
// the additions. Elements of mass 0 are left out of the top-p histograms: a bin of mass 0 is never the first
// to reach the goal.
//
// Bound: latency (barriers and dependent passes over shared memory); the traffic is 0.6 MB per row.
// Measured against 11 to 17 launches over a scratch in device memory, 151936 entries, us a call, before -> after:
//   top-k 20 top-p 0.95   1 row 57.7 -> 35.1   8 rows 70.9 -> 37.6   32 rows 133 -> 47.2   256 rows 956 -> 373
//   top-p 0.9             1 row 38.3 -> 35.5   8 rows 49.5 -> 41.0   32 rows 105 -> 55.5   256 rows 700 -> 407
//
//   * 8 CTAs of 512 threads: the largest cluster every device can place, and at 151936 entries two CTAs
//     (76 KB of row each) fit an SM, so 32 rows run at once.
//   * A shared-memory add on a 64-bit word is a compare-and-swap loop, and logits crowd into few of the
//     first level's bins. So masses are added as two 32-bit halves (16 + 17 bits; a slice has fewer than
//     65536 elements, so neither overflows), and top-k counts only what is at or above the bound of phase 1:
//     of g >= k disjoint groups of a row's elements the smallest group maximum has at least k elements at or
//     above it. Rows too long for shared memory are re-read from L2 and use 64-bit adds.
#include <cooperative_groups.h>

#include "kernels.h"
#include "nvfp4_ptx.cuh"
#include "sampling.cuh"

namespace nvfp4r {
namespace {

namespace cg = cooperative_groups;

constexpr int kCtas = 8;                       // CTAs per row
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kBins = 2048;
constexpr int kSeg = kBins / kCtas;            // bins that one CTA sums
constexpr int kMaxCached = 48 * 1024;          // elements of a slice kept in shared memory (192 KB)

__host__ __device__ constexpr int level_shift(int level) { return level == 0 ? 21 : (level == 1 ? 10 : 0); }
__host__ __device__ constexpr int level_bins(int level) { return level == 2 ? 1024 : 2048; }

__device__ __forceinline__ uint32_t warp_max_u(uint32_t v, int width) {
    for (int s = width / 2; s > 0; s >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, s));
    return v;
}

template <bool kCached>
__global__ void __launch_bounds__(kThreads, 2)
sample_truncated_kernel(const float* __restrict__ logits, int64_t row_stride, int V, int per, int top_k, float top_p,
                        unsigned long long seed, unsigned long long* __restrict__ draws,
                        int* __restrict__ last_ids, int* __restrict__ out) {
    extern __shared__ __align__(16) float s_row[];            // [per] when kCached
    // counts [kBins]; masses: low halves [kBins] and high halves [kBins], or 64-bit words [kBins]
    __shared__ __align__(16) uint32_t s_hist[2 * kBins];
    __shared__ unsigned long long s_scan[kSeg / 32];
    __shared__ float s_f[kWarps];
    __shared__ uint32_t s_u[kWarps];
    __shared__ int s_i[kWarps];
    // written by the CTAs of the cluster
    __shared__ float s_peer_max[kCtas];
    __shared__ uint32_t s_peer_bound[kCtas];
    __shared__ unsigned long long s_peer_total[kCtas];
    __shared__ unsigned long long s_pick_above;
    __shared__ uint32_t s_pick_bin;
    __shared__ float s_peer_best[kCtas];
    __shared__ int s_peer_arg[kCtas];

    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank());
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.y;
    pdl_launch_dependents();
    cluster.barrier_arrive();                                 // peers' shared memory may be written once all run
    for (int i = tid; i < 2 * kBins / 4; i += kThreads) reinterpret_cast<uint4*>(s_hist)[i] = make_uint4(0, 0, 0, 0);
    pdl_wait_prior();

    const float* row = logits + b * row_stride;
    const int lo = static_cast<int>(min(static_cast<int64_t>(rank) * per, static_cast<int64_t>(V)));
    const int len = min(per, V - lo);
    const int n4 = (len + 3) / 4;

    // ---- load, maximum ---------------------------------------------------------------------------
    float vmax = -INFINITY;                                   // fmaxf drops NaN
    if (kCached) {
        if ((reinterpret_cast<uintptr_t>(row + lo) & 15) == 0) {
            const float4* src = reinterpret_cast<const float4*>(row + lo);
            const int full = len / 4;
#pragma unroll 5
            for (int i = tid; i < full; i += kThreads) {
                const float4 v = __ldg(src + i);
                reinterpret_cast<float4*>(s_row)[i] = v;
                vmax = fmaxf(fmaxf(vmax, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
            }
            for (int i = full * 4 + tid; i < 4 * n4; i += kThreads) {
                const float v = i < len ? __ldg(row + lo + i) : -INFINITY;
                s_row[i] = v;
                vmax = fmaxf(vmax, v);
            }
        } else {
#pragma unroll 8
            for (int i = tid; i < 4 * n4; i += kThreads) {
                const float v = i < len ? __ldg(row + lo + i) : -INFINITY;
                s_row[i] = v;
                vmax = fmaxf(vmax, v);
            }
        }
    } else {
        for (int i = tid; i < len; i += kThreads) vmax = fmaxf(vmax, __ldg(row + lo + i));
    }
    // visits the slice's elements, the lower index first within a thread
    auto for_each = [&](auto&& f) {
        if (kCached) {
#pragma unroll 2
            for (int i = tid; i < n4; i += kThreads) {
                const float4 v = reinterpret_cast<const float4*>(s_row)[i];
                f(v.x, lo + 4 * i); f(v.y, lo + 4 * i + 1); f(v.z, lo + 4 * i + 2); f(v.w, lo + 4 * i + 3);
            }
        } else {
            for (int i = tid; i < len; i += kThreads) f(__ldg(row + lo + i), lo + i);
        }
    };

    // Bound of the k-th largest: groups of `width` threads, at least k of them in this CTA.
    const uint32_t my_key = sortable_key(vmax);
    int width = 32;
    while (width > 1 && kThreads / width < top_k) width >>= 1;
    uint32_t bound = 0u;
    if (top_k > 0 && top_k <= kThreads) {
        const uint32_t g = warp_max_u(my_key, width);
        bound = ~warp_max_u(~g, 32);                          // smallest of the warp's group maxima
    }
    float m = vmax;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if (lane == 0) { s_f[warp] = m; s_u[warp] = bound; }
    __syncthreads();
    cluster.barrier_wait();
    if (tid < kCtas) {
        float cm = s_f[0];
        uint32_t cb = s_u[0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) { cm = fmaxf(cm, s_f[w]); cb = min(cb, s_u[w]); }
        *cluster.map_shared_rank(&s_peer_max[rank], tid) = cm;
        *cluster.map_shared_rank(&s_peer_bound[rank], tid) = cb;
    }
    cluster.sync();
    m = s_peer_max[0];
    uint32_t floor_key = s_peer_bound[0];
#pragma unroll
    for (int q = 1; q < kCtas; ++q) { m = fmaxf(m, s_peer_max[q]); floor_key = max(floor_key, s_peer_bound[q]); }

    // ---- truncation --------------------------------------------------------------------------------
    uint32_t min_key = 0u, thr_key = 0u;                      // candidates / final set: key >= ...
#pragma unroll 1
    for (int mode = 0; mode < 2; ++mode) {                    // 0: top-k by count, 1: top-p by mass
        if (mode == 0 ? top_k <= 0 : !(top_p < 1.0f)) continue;
        const uint32_t skip_below = mode == 0 ? floor_key : min_key;
        uint32_t prefix = 0u;
        unsigned long long above = 0ull;                      // count / mass of the keys above the prefix
        unsigned long long goal = static_cast<unsigned long long>(top_k);
        bool all = false;
#pragma unroll 1
        for (int level = 0; level < 3; ++level) {
            const int shift = level_shift(level), prev_shift = level == 0 ? 31 : level_shift(level - 1);
            const uint32_t mask = static_cast<uint32_t>(level_bins(level) - 1);
            for_each([&](float x, int) {
                if (!(x > -INFINITY)) return;                 // -inf and NaN never enter the set
                const uint32_t key = sortable_key(x);
                if (key < skip_below) return;
                if (level > 0 && (key >> prev_shift) != prefix) return;
                const uint32_t bin = (key >> shift) & mask;
                if (mode == 0) {
                    atomicAdd(&s_hist[bin], 1u);
                    return;
                }
                // the maximum itself weighs exactly 2^32, also when it is +inf
                const unsigned long long w = x == m ? (1ull << 32) : __float2ull_rd(__expf(x - m) * 4294967296.0f);
                if (kCached) {
                    const uint32_t w_lo = static_cast<uint32_t>(w) & 0xffffu, w_hi = static_cast<uint32_t>(w >> 16);
                    if (w_lo != 0u) atomicAdd(&s_hist[bin], w_lo);
                    if (w_hi != 0u) atomicAdd(&s_hist[kBins + bin], w_hi);
                } else if (w != 0ull) {
                    atomicAdd(reinterpret_cast<unsigned long long*>(s_hist) + bin, w);
                }
            });
            cluster.sync();

            // this CTA's bins in descending order: thread t has bin kBins - 1 - (rank * kSeg + t)
            unsigned long long v = 0ull, incl = 0ull;
            const int bin = kBins - 1 - (rank * kSeg + tid);
            if (tid < kSeg) {
#pragma unroll
                for (int q = 0; q < kCtas; ++q) {
                    const uint32_t* h = cluster.map_shared_rank(s_hist, q);
                    if (mode == 0) v += h[bin];
                    else if (kCached) v += h[bin] + (static_cast<unsigned long long>(h[kBins + bin]) << 16);
                    else v += reinterpret_cast<const unsigned long long*>(h)[bin];
                }
                incl = v;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const unsigned long long o = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += o;
                }
                if (lane == 31) s_scan[warp] = incl;
            }
            __syncthreads();
            unsigned long long seg = 0ull;
#pragma unroll
            for (int w = 0; w < kSeg / 32; ++w) {
                if (w < warp) incl += s_scan[w];
                seg += s_scan[w];
            }
            if (tid < kCtas) *cluster.map_shared_rank(&s_peer_total[rank], tid) = seg;
            cluster.sync();

            unsigned long long total = 0ull, base = 0ull;
#pragma unroll
            for (int q = 0; q < kCtas; ++q) {
                if (q < rank) base += s_peer_total[q];
                total += s_peer_total[q];
            }
            if (mode == 1 && level == 0) {
                // candidate set = everything counted here (the top-k set when top-k ran before)
                goal = static_cast<unsigned long long>(ceil(static_cast<double>(top_p) * static_cast<double>(total)));
                if (goal < 1ull) goal = 1ull;
            }
            for (int i = tid; i < 2 * kBins / 4; i += kThreads)
                reinterpret_cast<uint4*>(s_hist)[i] = make_uint4(0, 0, 0, 0);
            all = above + total < goal;                       // same decision in every thread of the cluster
            if (all) break;
            const unsigned long long through = above + base + incl;
            if (tid < kSeg && through >= goal && through - v < goal) {
#pragma unroll
                for (int q = 0; q < kCtas; ++q) {
                    *cluster.map_shared_rank(&s_pick_bin, q) = static_cast<uint32_t>(bin);
                    *cluster.map_shared_rank(&s_pick_above, q) = through - v;
                }
            }
            cluster.sync();
            prefix = (level == 0 ? 0u : prefix << (level == 2 ? 10 : 11)) | s_pick_bin;
            above = s_pick_above;
        }
        // the goal is never reached (fewer finite candidates than k): everything that is left stays
        thr_key = all ? min_key : prefix;
        min_key = thr_key;
        __syncthreads();                                      // histogram zeroed before the next descent adds to it
    }

    // ---- Gumbel-max draw within the set --------------------------------------------------------------
    const unsigned long long key = gumbel_key(seed, b, draws[b]);
    float best = -INFINITY;
    int arg = 0x7fffffff;
    for_each([&](float x, int i) {
        if (!(x > -INFINITY) || sortable_key(x) < thr_key) return;
        const float s = x + gumbel_noise(key, i);
        if (s > best) { best = s; arg = i; }
    });
    auto take = [&](float ob, int oa) {
        if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
    };
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, s);
        take(ob, __shfl_xor_sync(0xffffffffu, arg, s));
    }
    if (lane == 0) { s_f[warp] = best; s_i[warp] = arg; }
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int w = 1; w < kWarps; ++w) take(s_f[w], s_i[w]);
        *cluster.map_shared_rank(&s_peer_best[rank], 0) = best;
        *cluster.map_shared_rank(&s_peer_arg[rank], 0) = arg;
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
#pragma unroll
        for (int q = 0; q < kCtas; ++q) take(s_peer_best[q], s_peer_arg[q]);
        // a row without any finite candidate (all -inf or NaN) yields id 0, never the sentinel
        if (arg == 0x7fffffff) arg = 0;
        out[b] = arg;
        draws[b] += 1ull;
        if (last_ids != nullptr) {
            last_ids[2 * b] = last_ids[2 * b + 1];
            last_ids[2 * b + 1] = arg;
        }
    }
}

}  // namespace

cudaError_t launch_sample_truncated(const float* logits, int64_t row_stride, int B, int V, int top_k, float top_p,
                                    unsigned long long seed, unsigned long long* draws, int* last_ids, int* out,
                                    cudaStream_t stream) {
    const int per = static_cast<int>(((static_cast<int64_t>(V) + kCtas - 1) / kCtas + 3) / 4 * 4);
    const bool cached = per <= kMaxCached;
    static bool attr_done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (cached && (dev < 0 || dev >= 64 || !attr_done[dev])) {
        e = cudaFuncSetAttribute(sample_truncated_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kMaxCached * static_cast<int>(sizeof(float)));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kCtas, static_cast<unsigned>(B));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = cached ? static_cast<size_t>(per) * sizeof(float) : 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kCtas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gemv_tuning().use_pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, cached ? sample_truncated_kernel<true> : sample_truncated_kernel<false>, logits,
                              row_stride, V, per, top_k, top_p, seed, draws, last_ids, out);
}

}  // namespace nvfp4r
