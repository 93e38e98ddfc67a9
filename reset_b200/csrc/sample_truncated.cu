// Top-k / top-p sampling of one id per row in one launch: one thread-block cluster of eight (or sixteen) CTAs per row.
//
// The row is read from memory once; each CTA keeps its share of it in shared memory and all exchange
// histograms, totals and picks through distributed shared memory with cluster barriers. Phases:
//   1. load, row maximum;
//   2. top-k up to 128: the k-th largest of the 128 warps' maxima bounds the k-th largest value from below (k
//      groups have an element at or above it). What reaches the bound goes to one CTA's list, a few more than k
//      on unordered logits; with at most 512 entries that CTA settles the row by comparing all pairs, one
//      entry per thread, and the launch ends;
//   3. otherwise, per truncation (top-k by count, then top-p by mass) one histogram of 2048 equal steps of the distance to
//      the row maximum, 22.2 in all by mass (what lies further has none), 89 by count: the CTA whose bins cross the goal announces the
//      bin, its entries go to one CTA's list, and with at most 512 of them that CTA finds the threshold by comparing all
//      pairs. The distance rounds monotonically, so bins are in the order of the values;
//   4. where more entries share the bin, or the goal lies beyond the steps, a radix descent over the order-preserving keys,
//      11 + 11 + 10 bits: histogram of the keys that share the prefix found so far, each CTA sums its share of the
//      2048 bins over all histograms, and the CTA whose bins cross the goal announces the bin. After
//      the last level the prefix is the key of the last token kept; equal keys are all kept;
//   5. arg-max of logit + Gumbel noise among the keys at or above the threshold.
// Mass is exp(x - row max) scaled by 2^32 and truncated to an integer, so no result depends on the order of
// the additions. Elements of mass 0 are left out of the top-p histograms: a bin of mass 0 is never the first
// to reach the goal.
//
// Bound: latency (barriers and dependent passes over shared memory); the traffic is 0.6 MB per row.
// Measured, 151936 entries. Top-k 20 top-p 0.95, us a call, 11 to 17 launches over a scratch in device memory -> one launch
// (and that without phase 2): 1 row 57.7 -> 7.4 (35.1), 8 rows 70.9 -> 8.4 (37.6), 32 rows 133 -> 10.1 (47.2), 256 rows
// 956 -> 90 (373). Larger sets, device us in a CUDA graph with the counters' reset, radix descent alone -> phase 3, the masses in
// 32-bit halves and the draw's logarithms only where they can matter:
//   top-p 0.9   1 row 31.6 -> 19.1   8 rows 39.4 -> 26.7   32 rows 53.8 -> 38.7     top-k 1000, 8 rows 27.9 -> 22.4
//   top-k 150 top-p 0.8, 8 rows 40.2 -> 28.6
// of which, 8 rows in clusters of eight, thousand clocks: load 5, histogram 11, its bin 6, list 5, pairs 3, draw 13.
//
//   * 8 CTAs of 512 threads (16 for a few rows of top-p alone, where the device can place them): the largest cluster every
//     device can place, and at 151936 entries two CTAs
//     (76 KB of row each) fit an SM, so 32 rows run at once.
//   * A shared-memory add on a 64-bit word is a compare-and-swap loop, and logits crowd into few of the
//     first level's bins. So masses are added as two 32-bit halves (16 + 17 bits; a slice has fewer than
//     65536 elements, so neither overflows), and top-k counts only what reaches the bound of phase 2. Rows too
//     long for shared memory are re-read from L2 and use 64-bit adds.
#include <cooperative_groups.h>

#include <atomic>

#include "kernels.h"
#include "nvfp4_ptx.cuh"
#include "sampling.cuh"

namespace nvfp4r {
namespace {

namespace cg = cooperative_groups;

constexpr int kFewCtas = 8, kMostCtas = 16;    // CTAs per row
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kBins = 2048;
constexpr int kMaxCached = 48 * 1024;          // elements of a slice kept in shared memory (192 KB)

__host__ __device__ constexpr int level_shift(int level) { return level == 0 ? 21 : (level == 1 ? 10 : 0); }
__host__ __device__ constexpr int level_bins(int level) { return level == 2 ? 1024 : 2048; }

constexpr int kGroups = kFewCtas * kWarps;     // groups of a row for phase 2: one per warp
constexpr int kListMax = kThreads;                // candidates that one CTA settles, one per thread

__device__ __forceinline__ unsigned long long mass_of(float x, float m) {
    // the maximum itself weighs exactly 2^32, also when it is +inf
    return x == m ? (1ull << 32) : __float2ull_rd(__expf(x - m) * 4294967296.0f);
}

// The same number in two halves of 16 and 17 bits: powers of two and differences are exact, so no 64-bit conversion.
__device__ __forceinline__ void mass_halves(float x, float m, uint32_t& w_lo, uint32_t& w_hi) {
    const float t = x == m ? 65536.0f : __expf(x - m) * 65536.0f;
    w_hi = static_cast<uint32_t>(t);
    w_lo = static_cast<uint32_t>((t - static_cast<float>(w_hi)) * 65536.0f);
}

// kFew: 0 < top_k <= kGroups (its own instance: the list's code costs the descent registers)
template <bool kCached, bool kFew, int kCtas>
__global__ void __launch_bounds__(kThreads, 2)
sample_truncated_kernel(const float* __restrict__ logits, int64_t row_stride, int V, int per, int top_k, float top_p,
                        unsigned long long seed, unsigned long long* __restrict__ draws,
                        int* __restrict__ last_ids, int* __restrict__ out) {
    constexpr int kSeg = kBins / kCtas;                       // bins that one CTA sums
    static_assert(!kFew || kCtas == kFewCtas, "one group per warp of eight CTAs");
    extern __shared__ __align__(16) float s_row[];            // [per] when kCached
    // counts [kBins]; masses: low halves [kBins] and high halves [kBins], or 64-bit words [kBins]
    __shared__ __align__(16) uint32_t s_hist[2 * kBins];
    __shared__ unsigned long long s_scan[kSeg / 32];
    __shared__ float s_f[kWarps];
    __shared__ int s_i[kWarps];
    // written by the CTAs of the cluster
    __shared__ float s_peer_max[kCtas];
    __shared__ uint32_t s_group[kGroups];
    __shared__ uint32_t s_bound;
    __shared__ int s_count;                                   // rank 0: candidates of the row
    __shared__ float s_list_x[kListMax];
    __shared__ int s_list_i[kListMax];
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

    float m = vmax;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if (lane == 0) s_f[warp] = m;
    if (tid == 0) s_count = 0;
    __syncthreads();
    cluster.barrier_wait();
    if (kFew && tid < kGroups)                                // 16 group maxima to each of 8 CTAs
        *cluster.map_shared_rank(&s_group[rank * kWarps + tid % kWarps], tid / kWarps) = sortable_key(s_f[tid % kWarps]);
    if (tid < kCtas) {
        float cm = s_f[0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) cm = fmaxf(cm, s_f[w]);
        *cluster.map_shared_rank(&s_peer_max[rank], tid) = cm;
    }
    cluster.sync();
    m = s_peer_max[0];
#pragma unroll
    for (int q = 1; q < kCtas; ++q) m = fmaxf(m, s_peer_max[q]);

    // ---- few candidates: one CTA settles the row ---------------------------------------------------
    uint32_t floor_key = 0u;
    bool settled = false;
    if (kFew) {
        if (tid < kGroups) {
            const uint32_t mine = s_group[tid];
            int r = 0;
            for (int j = 0; j < kGroups; ++j) r += s_group[j] > mine || (s_group[j] == mine && j < tid);
            if (r == top_k - 1) s_bound = mine;
        }
        __syncthreads();
        floor_key = s_bound;
        int* count = cluster.map_shared_rank(&s_count, 0);
        float* list_x = cluster.map_shared_rank(s_list_x, 0);
        int* list_i = cluster.map_shared_rank(s_list_i, 0);
        for_each([&](float x, int i) {
            if (!(x > -INFINITY) || sortable_key(x) < floor_key) return;
            const int at = atomicAdd(count, 1);
            if (at < kListMax) { list_x[at] = x; list_i[at] = i; }
        });
        cluster.sync();
        settled = *count <= kListMax;                            // same answer in every thread of the cluster
    }
    float best = -INFINITY;
    int arg = 0x7fffffff;
    auto take = [&](float ob, int oa) {
        if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
    };
    auto block_best = [&] {                                   // thread 0 ends up with the CTA's
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, s);
            take(ob, __shfl_xor_sync(0xffffffffu, arg, s));
        }
        if (lane == 0) { s_f[warp] = best; s_i[warp] = arg; }
        __syncthreads();
        if (tid == 0)
#pragma unroll
            for (int w = 1; w < kWarps; ++w) take(s_f[w], s_i[w]);
    };
    auto finish = [&] {
        // a row without any finite candidate (all -inf or NaN) yields id 0, never the sentinel
        if (arg == 0x7fffffff) arg = 0;
        out[b] = arg;
        draws[b] += 1ull;
        if (last_ids != nullptr) {
            last_ids[2 * b] = last_ids[2 * b + 1];
            last_ids[2 * b + 1] = arg;
        }
    };
    if (kFew && settled) {
        if (rank == 0) {
            // a candidate stays when fewer than k are larger, and when what is larger and stays by count has
            // less than the goal's mass
            const int n = s_count;
            const bool have = tid < n;
            const float x = have ? s_list_x[tid] : 0.0f;
            const uint32_t mine = have ? sortable_key(x) : 0u;
            uint32_t* keys = s_hist;                          // [kListMax]
            unsigned long long* mass = reinterpret_cast<unsigned long long*>(s_hist + kListMax);      // [kListMax]
            keys[tid] = mine;
            __syncthreads();
            bool keep = have;
            if (have) {
                int larger = 0;
                for (int j = 0; j < n; ++j) larger += keys[j] > mine;
                keep = larger < top_k;
            }
            if (top_p < 1.0f) {
                mass[tid] = keep ? mass_of(x, m) : 0ull;
                __syncthreads();
                if (keep) {
                    unsigned long long total = 0ull, above = 0ull;
                    for (int j = 0; j < n; ++j) {
                        const unsigned long long w = mass[j];
                        total += w;
                        if (keys[j] > mine) above += w;
                    }
                    unsigned long long goal =
                        static_cast<unsigned long long>(ceil(static_cast<double>(top_p) * static_cast<double>(total)));
                    if (goal < 1ull) goal = 1ull;
                    keep = above < goal;
                }
            }
            const unsigned long long key = gumbel_key(seed, b, draws[b]);
            if (keep) { best = x + gumbel_noise(key, s_list_i[tid]); arg = s_list_i[tid]; }
            if (best == -INFINITY) arg = 0x7fffffff;
            block_best();
            if (tid == 0) finish();
        }
        cluster.sync();                                       // rank 0's count has been read by all
        return;
    }

    // ---- truncation --------------------------------------------------------------------------------
    // Sum of the bins, in descending order of the values, up to the one that crosses the goal; called by all threads
    // of the cluster behind a histogram. False: the bins do not reach the goal. The histogram is cleared.
    auto find_bin = [&](int mode, unsigned long long above, unsigned long long& goal, bool first) {
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
        if (mode == 1 && first) {
            // candidate set = everything counted here (the top-k set when top-k ran before)
            goal = static_cast<unsigned long long>(ceil(static_cast<double>(top_p) * static_cast<double>(total)));
            if (goal < 1ull) goal = 1ull;
        }
        for (int i = tid; i < 2 * kBins / 4; i += kThreads)
            reinterpret_cast<uint4*>(s_hist)[i] = make_uint4(0, 0, 0, 0);
        if (tid == 0) s_count = 0;                            // (rank 0's is the one in use)
        if (above + total < goal) return false;               // same decision in every thread of the cluster
        const unsigned long long through = above + base + incl;
        if (tid < kSeg && through >= goal && through - v < goal) {
#pragma unroll
            for (int q = 0; q < kCtas; ++q) {
                *cluster.map_shared_rank(&s_pick_bin, q) = static_cast<uint32_t>(bin);
                *cluster.map_shared_rank(&s_pick_above, q) = through - v;
            }
        }
        cluster.sync();
        return true;
    };
    auto add_mass = [&](uint32_t bin, float x) {
        if (kCached) {
            uint32_t w_lo, w_hi;
            mass_halves(x, m, w_lo, w_hi);
            if (w_lo != 0u) atomicAdd(&s_hist[bin], w_lo);
            if (w_hi != 0u) atomicAdd(&s_hist[kBins + bin], w_hi);
        } else {
            const unsigned long long w = mass_of(x, m);
            if (w != 0ull) atomicAdd(reinterpret_cast<unsigned long long*>(s_hist) + bin, w);
        }
    };
    // bin 2047: the maximum; bin 0: everything beyond the steps, at a distance of 22.2 by mass, 89 by count
    auto step_bin = [&](float x, int mode) {
        return static_cast<uint32_t>(kBins - 1) -
               (x == m ? 0u : static_cast<uint32_t>(fminf((m - x) * (mode == 0 ? 23.0f : 92.0f), static_cast<float>(kBins - 1))));
    };
    uint32_t min_key = 0u, thr_key = 0u;                      // candidates / final set: key >= ...
#pragma unroll 1
    for (int mode = 0; mode < 2; ++mode) {                    // 0: top-k by count, 1: top-p by mass
        if (mode == 0 ? top_k <= 0 : !(top_p < 1.0f)) continue;
        const uint32_t skip_below = mode == 0 ? floor_key : min_key;
        uint32_t prefix = 0u;
        unsigned long long above = 0ull;                      // count / mass of the keys above the prefix
        unsigned long long goal = static_cast<unsigned long long>(top_k);
        bool all = false;

        for_each([&](float x, int) {
            if (!(x > -INFINITY) || sortable_key(x) < skip_below) return;      // -inf and NaN never enter the set
            if (mode == 0) atomicAdd(&s_hist[step_bin(x, mode)], 1u);
            else if (!(m - x > 22.25f)) add_mass(step_bin(x, mode), x);       // beyond: less than 2^-32, no mass
        });
        if (!find_bin(mode, 0ull, goal, true)) {
            all = true;
        } else if (s_pick_bin != 0u) {
            const uint32_t pick = s_pick_bin;
            int* count = cluster.map_shared_rank(&s_count, 0);
            float* list_x = cluster.map_shared_rank(s_list_x, 0);
            const float step = mode == 0 ? 23.0f : 92.0f, first = static_cast<float>(kBins - 1 - static_cast<int>(pick));
            for_each([&](float x, int) {
                const float d = x == m ? 0.0f : (m - x) * step;      // step_bin(x, mode) == pick; false for NaN
                if (!(d >= first && d < first + 1.0f) || sortable_key(x) < skip_below) return;
                const int at = atomicAdd(count, 1);
                if (at < kListMax) list_x[at] = x;
            });
            cluster.sync();
            const int n = *count;
            if (n <= kListMax) {                              // same answer in every thread of the cluster
                if (rank == 0) {
                    // an entry stays while what is larger is less than the goal; the smallest that stays is the threshold
                    const bool have = tid < n;
                    const float x = have ? s_list_x[tid] : 0.0f;
                    const uint32_t mine = have ? sortable_key(x) : 0u;
                    if (tid == 0) s_bound = 0xffffffffu;
                    unsigned long long* weight = reinterpret_cast<unsigned long long*>(s_hist + kListMax);
                    s_hist[tid] = mine;
                    weight[tid] = have ? (mode == 0 ? 1ull : mass_of(x, m)) : 0ull;
                    __syncthreads();
                    if (have) {
                        unsigned long long larger = s_pick_above;
                        for (int j = 0; j < n; ++j)
                            if (s_hist[j] > mine) larger += weight[j];
                        if (larger < goal) atomicMin(&s_bound, mine);
                    }
                    __syncthreads();
                    if (tid < kCtas) *cluster.map_shared_rank(&s_pick_bin, tid) = s_bound;
                    for (int i = tid; i < 3 * kListMax; i += kThreads) s_hist[i] = 0u;
                }
                cluster.sync();
                thr_key = min_key = s_pick_bin;
                continue;
            }
        }
#pragma unroll 1
        for (int level = 0; level < 3 && !all; ++level) {
            const int shift = level_shift(level), prev_shift = level == 0 ? 31 : level_shift(level - 1);
            const uint32_t mask = static_cast<uint32_t>(level_bins(level) - 1);
            for_each([&](float x, int) {
                if (!(x > -INFINITY)) return;
                const uint32_t key = sortable_key(x);
                if (key < skip_below) return;
                if (level > 0 && (key >> prev_shift) != prefix) return;
                const uint32_t bin = (key >> shift) & mask;
                if (mode == 0) atomicAdd(&s_hist[bin], 1u);
                else add_mass(bin, x);
            });
            if (!find_bin(mode, above, goal, false)) {
                all = true;
                break;
            }
            prefix = (level == 0 ? 0u : prefix << (level == 2 ? 10 : 11)) | s_pick_bin;
            above = s_pick_above;
        }
        // the goal is never reached (fewer finite candidates than k): everything that is left stays
        thr_key = all ? min_key : prefix;
        min_key = thr_key;
        __syncthreads();                                      // histogram zeroed before the next descent adds to it
    }

    // ---- Gumbel-max draw within the set --------------------------------------------------------------
    // The two logarithms are taken only where they can matter: -log(-log u) <= -log(1 - u), so an element stays below
    // the best score of the CTA so far when 1 - u > exp(x - best). The 1 % covers the rounding of the two sides; the sum
    // x + noise rounds up by half a unit of best at most, which 2^-23 best in the exponent covers at any magnitude.
    const unsigned long long key = gumbel_key(seed, b, draws[b]);
    if (tid == 0) s_bound = 0u;
    __syncthreads();
    volatile uint32_t* bound = &s_bound;                      // the CTA's best score, as a key
    for_each([&](float x, int i) {
        if (!(x > -INFINITY) || sortable_key(x) < thr_key) return;
        const float u = gumbel_uniform(key, i);
        const uint32_t so_far = *bound;
        const float top = key_value(so_far);
        if (so_far != 0u && 1.0f - u > 1.01f * __expf(fmaf(fabsf(top), 1.0f / 8388608.0f, x - top))) return;
        const float s = x + gumbel_of(u);
        if (s > best) { best = s; arg = i; }
        const uint32_t mine = sortable_key(s);
        if (mine > so_far) atomicMax(&s_bound, mine);
    });
    block_best();
    if (tid == 0) {
        *cluster.map_shared_rank(&s_peer_best[rank], 0) = best;
        *cluster.map_shared_rank(&s_peer_arg[rank], 0) = arg;
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
#pragma unroll
        for (int q = 0; q < kCtas; ++q) take(s_peer_best[q], s_peer_arg[q]);
        finish();
    }
}

// Rows that clusters of 16 CTAs (more than every device can place) can have at once: asked once per device for slices that
// leave room for two CTAs per SM and once for the largest.
int rows_at_once(int dev, int per) {
    if (dev < 0 || dev >= 64) return 0;
    constexpr int kTwoPerSm = 22 * 1024;
    static std::atomic<int> known[64][2] = {};                // answer + 1
    const int large = per > kTwoPerSm;
    const int last = known[dev][large].load(std::memory_order_acquire);
    if (last > 0) return last - 1;
    const auto kern = sample_truncated_kernel<true, false, kMostCtas>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kMostCtas, 1);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(large ? kMaxCached : kTwoPerSm) * sizeof(float);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kMostCtas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxCached * static_cast<int>(sizeof(float))) != cudaSuccess ||
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
    }
    known[dev][large].store(n + 1, std::memory_order_release);
    return n;
}

}  // namespace

cudaError_t launch_sample_truncated(const float* logits, int64_t row_stride, int B, int V, int top_k, float top_p,
                                    unsigned long long seed, unsigned long long* draws, int* last_ids, int* out,
                                    cudaStream_t stream) {
    const bool few = top_k > 0 && top_k <= kGroups;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const auto slice = [&](int ctas) { return static_cast<int>(((static_cast<int64_t>(V) + ctas - 1) / ctas + 3) / 4 * 4); };
    // Top-p alone is passes over the row: sixteen CTAs, while all rows find a place at once. 1 row 23.0 -> 19.2 us, 4 rows
    // 29.8 -> 23.4, 8 rows 30.0 -> 26.8, 12 rows 30.4 -> 29.0. With top-k the row is counted in less time than the larger
    // cluster's barriers add: 8 rows, top-k 1000 22.3 / 23.7, top-k 150 top-p 0.8 28.5 / 30.3.
    const bool most = top_k <= 0 && slice(kMostCtas) <= kMaxCached && B <= rows_at_once(dev, slice(kMostCtas));
    const int ctas = most ? kMostCtas : kFewCtas, per = slice(ctas);
    const bool cached = per <= kMaxCached;
    const auto kern = most ? sample_truncated_kernel<true, false, kMostCtas>
                      : cached ? (few ? sample_truncated_kernel<true, true, kFewCtas> : sample_truncated_kernel<true, false, kFewCtas>)
                               : (few ? sample_truncated_kernel<false, true, kFewCtas> : sample_truncated_kernel<false, false, kFewCtas>);
    static bool attr_done[2][64] = {};
    if (!most && cached && (dev < 0 || dev >= 64 || !attr_done[few][dev])) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxCached * static_cast<int>(sizeof(float)));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[few][dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas), static_cast<unsigned>(B));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = cached ? static_cast<size_t>(per) * sizeof(float) : 0;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gemv_tuning().use_pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, logits, row_stride, V, per, top_k, top_p, seed, draws, last_ids, out);
}

}  // namespace nvfp4r
