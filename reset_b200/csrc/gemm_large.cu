// NVFP4 W4A4 GEMM on the 5th-generation tensor cores for more tokens than a decode launch takes
// (sm_100a): out[m, n] = alpha * sum_k dq(W[n, k]) * dq(X[m, k]).
//
// The decode kernels (linear_packed.cu, gemm_tcgen05.cu) take at most 32 tokens per launch, keep the
// tokens of a K part in shared memory and stream the whole weight once per launch: M tokens cost
// M / 32 passes over the weight and M / 32 quantizations of the same token by every CTA. Here one
// launch takes all tokens: a tile is 128 weight rows x bn tokens (bn = 16 .. 256), both operands
// are staged through one ring, and the weight tile is re-used for bn tokens.
//
//   A operand  128 weight rows   (TMEM lanes of the accumulator)
//   B operand  bn tokens         (TMEM columns)
//
// Operands come in one of two forms (template parameter kTma):
//   packed     weight in the packed block format of linear_packed.cu (18 432 contiguous bytes per
//              128 rows x 256 K), tokens written by quant_pack_kernel in the same kind of block for
//              bn rows: [bn x 128 B of codes, 128-byte swizzle][2048 B of scales per 128 rows].
//              A pipeline stage (256 K-elements) is two 1-D bulk copies.
//   row-major  codes through 2-D tensor maps (128-byte swizzle), scales in the 128x4-tiled layout as
//              512-byte chunks: the operands of the raw gemm operator.
//
// Persistent CTAs, one per SM, ten warps: warp 0 producer, warp 1 MMA issuer, warps 2-9 epilogue (two
// per TMEM lane quadrant, each half of the columns). Schedule: CTA c first computes whole tiles c, c + G, ...
// for `dp_rounds` rounds; the K blocks of the tiles that are left, laid end to end, are then cut into one
// equal range for each of `sk_ctas` CTAs (stream-K). A tile that two or more CTAs share is summed from
// fp32 partials, in K order, by the one that finishes last (atomic ticket; nothing waits, results do not
// depend on the order of arrival).
//
// What bounds it: the bytes that one SM takes in from L2. A stage of 128 x 256 x 256 K is 55 KB for 512 clocks of MMA,
// 107 bytes per clock; profiled on 24576x4096 with 2048 tokens it takes in 60 (1.36 GB in 104 us), the tensor
// pipe is busy for 56 % of the active clocks and DRAM for 17 % of the time. So the time is stages x bytes / that rate:
// hence the widest tile that still fills the SMs. The MMA issuer is straight-line code per K block: rolled loops made
// each tcgen05 instruction wait for its operands (same call, quantizer included: 111 -> 102 us in a burst at 1965 MHz,
// 4.0 PFLOP/s; calls kept up for seconds settle at 122 us, 1515 MHz under the power cap).
// Measured, one call: 24576x4096 with 2048 tokens 2994 -> 121 us, 6144x4096 with 333 tokens 158 -> 13.7 us,
// 10240x5120 with 45 tokens 35.5 -> 12.6 us; nvfp4r.quant + nvfp4r.gemm 4096x12288 with 128 tokens 147 ->
// 22.5 us (left: 32 tokens per pass).
#include <cuda.h>

#include <atomic>
#include <mutex>

#include "kernels.h"
#include "quant_core.cuh"
#include "status_mirror.cuh"
#include "tcgen05_ptx.cuh"

namespace nvfp4r {
namespace {

using namespace tc;

constexpr int kRows = 128;                           // weight rows of a tile
constexpr int kBK = 256;                             // K elements per stage
constexpr int kABytes = kRows * 128 + 2048;          // codes + scales of the weight block
constexpr int kACodes = kRows * 128;
constexpr int kMaxStagesL = 8;
constexpr int kEpiWarps = 8;
constexpr int kThreadsL = (2 + kEpiWarps) * 32;
constexpr int kSmemBudget = 225 * 1024;              // dynamic part, 1 KB of it for alignment
// Time model of plan_large, nanoseconds, fitted to sweeps over tile widths and both schedules (eight weights,
// 16 .. 2048 tokens): a stage costs 200 ns + 1.3 ns per token of the tile; sharing a tile costs 2 us (partial
// stores, fence, ticket) and 0.7 us per part and 64 columns (one trip to L2 each).
constexpr double kStageBase = 200.0, kStagePerToken = 1.3, kFixBase = 2000.0, kFixPerPart = 700.0;
constexpr uint32_t kTmemColsL = 512;
constexpr uint32_t kColSfaL = 256, kColSfbL = 288;   // two buffers of 16, two of 32 columns

struct alignas(64) LargeParams {
    CUtensorMap map_w, map_x;                        // row-major form only
    const uint8_t* w;                                // packed weight blocks
    const uint8_t* x;                                // packed token blocks
    const uint8_t* wsf;                              // row-major form: 128x4-tiled scales
    const uint8_t* xsf;
    void* out;
    int64_t ldc;
    int M, N, bn, nch, tiles, tiles_m, kblocks, k64; // nch = 128-row scale chunks per token tile
    int stages;
    int dp_rounds, sk_base, sk_ctas, sk_q, sk_r;     // stream-K from tile sk_base on: sk_q (+1 for the first sk_r) K blocks per CTA
    float alpha;
    float* partials;                                 // [2 * sk_ctas][bn / 4][128][4]
    unsigned* tickets;                               // [tiles], zero before the launch, left zero
};

__device__ int g_large_status = 0;

// ---- token quantizer -------------------------------------------------------------------------
// One thread per 16-element block; four lanes share one 32-bit store of scales. Also clears the
// tickets of the GEMM that follows.
__global__ void __launch_bounds__(256)
quant_pack_kernel(const __nv_bfloat16* __restrict__ x, int64_t x_row_stride, int K, const float* __restrict__ gs_ptr,
                  bool exact, uint8_t* __restrict__ packed, int bn, int nch, int kblocks,
                  unsigned* __restrict__ tickets, int n_tickets) {
    pdl_launch_dependents();
    const int row = blockIdx.x;
    const int mt = row / bn, r = row - mt * bn;
    const int col = blockIdx.y * 256 + threadIdx.x;
    const float gs = __ldg(gs_ptr);
    const QuantScales q = exact ? make_quant_scales<kRcpExact>(gs) : make_quant_scales<kRcpApprox>(gs);
    pdl_wait_prior();
    if (blockIdx.y == 0)
        for (int i = row * 256 + threadIdx.x; i < n_tickets; i += gridDim.x * 256) tickets[i] = 0u;
    if (col >= K / kBlockElems) return;               // K % 128 == 0: groups of eight lanes leave together
    const uint4* src = reinterpret_cast<const uint4*>(x + row * x_row_stride + static_cast<int64_t>(col) * kBlockElems);
    const uint4 lo = __ldg(src), hi = __ldg(src + 1);
    uint32_t c[2];
    const uint32_t sf = quantize_block16_rt(lo, hi, q, exact, c);
    const int kb = col >> 4, b = col & 15;
    uint8_t* base = packed + (static_cast<int64_t>(mt) * kblocks + kb) * (bn * 128 + nch * 2048);
    *reinterpret_cast<uint2*>(base + swz128(r, b * 8)) = make_uint2(c[0], c[1]);
    const unsigned live = __activemask();
    uint32_t s4 = sf << (8 * (b & 3));
    s4 |= __shfl_xor_sync(live, s4, 1);
    s4 |= __shfl_xor_sync(live, s4, 2);
    if ((b & 3) == 0)
        *reinterpret_cast<uint32_t*>(base + bn * 128 + (r >> 7) * 2048 + (b >> 2) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4) = s4;
}

// ---- work of one CTA -------------------------------------------------------------------------
struct Segment { int tile, k0, k1; };

struct Walker {
    int round = 0, cur, end;
    __device__ __forceinline__ explicit Walker(const LargeParams& p) {
        const int c = blockIdx.x;
        cur = c * p.sk_q + min(c, p.sk_r);
        end = c < p.sk_ctas ? cur + p.sk_q + (c < p.sk_r ? 1 : 0) : cur;
    }
    __device__ __forceinline__ bool next(const LargeParams& p, Segment& s) {
        if (round < p.dp_rounds) {
            s.tile = blockIdx.x + round * gridDim.x;
            ++round;
            s.k0 = 0;
            s.k1 = p.kblocks;
            return s.tile < p.tiles;
        }
        if (cur >= end) return false;
        const int t = cur / p.kblocks;
        s.tile = p.sk_base + t;
        s.k0 = cur - t * p.kblocks;
        s.k1 = min(p.kblocks, s.k0 + end - cur);
        cur += s.k1 - s.k0;
        return true;
    }
};

// Position of a K block in the stream-K sequence -> the CTA whose range holds it; first position of CTA c.
__device__ __forceinline__ int sk_owner(const LargeParams& p, int i) {
    const int head = p.sk_r * (p.sk_q + 1);
    return i < head ? i / (p.sk_q + 1) : p.sk_r + (i - head) / p.sk_q;
}
__device__ __forceinline__ int sk_start(const LargeParams& p, int c) { return c * p.sk_q + min(c, p.sk_r); }

// One K block: the scale copies first, so that no MMA waits behind its own copy. Straight-line code with
// compile-time counts: with rolled loops every instruction waits for its operands to reach uniform registers.
template <int kChunks>
__device__ __forceinline__ void issue_block(uint32_t d, uint64_t a, uint64_t b, uint64_t sa, uint64_t sb, uint32_t idesc,
                                            uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        tc_cp_scales(sfa + 4 * k, sa + 32 * k);
#pragma unroll
        for (int j = 0; j < kChunks; ++j) tc_cp_scales(sfb + 4 * kChunks * k + 4 * j, sb + 128 * j + 32 * k);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        tc_mma_nvf4(d, a + 2 * k, b + 2 * k, idesc, sfa + 4 * k, sfb + 4 * kChunks * k, k == 0 ? accumulate : 1u);
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

template <int kDtype>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    if (kDtype == 0) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Store 16 accumulator columns (tokens m0 .. m0+15) of this lane's weight row n.
// M-major 16-bit: neighbouring lanes hold neighbouring n, so a pair of lanes trades halves and every
// store is 4 bytes: 16 lanes x 4 B for token m from the even lanes, the same for m + 1 from the odd.
template <int kDtype, bool kNMajor>
__device__ __forceinline__ void store16(const LargeParams& p, int n, int m0, const float v[16], int lane, bool vec) {
    const float al = p.alpha;
    if (kNMajor) {
        if (kDtype == 2) {
            float* o = static_cast<float*>(p.out) + static_cast<int64_t>(n) * p.ldc + m0;
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (m0 + j < p.M) o[j] = v[j] * al;
        } else {
            uint16_t* o = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(n) * p.ldc + m0;
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) w[j] = pack2<kDtype>(v[2 * j] * al, v[2 * j + 1] * al);
            if (vec && m0 + 16 <= p.M) {
                reinterpret_cast<uint4*>(o)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                reinterpret_cast<uint4*>(o)[1] = make_uint4(w[4], w[5], w[6], w[7]);
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (m0 + j < p.M) o[j] = static_cast<uint16_t>(j & 1 ? w[j >> 1] >> 16 : w[j >> 1]);
            }
        }
    } else if (kDtype == 2) {
        float* o = static_cast<float*>(p.out) + static_cast<int64_t>(m0) * p.ldc + n;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (m0 + j < p.M) o[static_cast<int64_t>(j) * p.ldc] = v[j] * al;
    } else {
        const bool odd = lane & 1;
        uint16_t* o = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(m0 + (odd ? 1 : 0)) * p.ldc + (n & ~1);
        const int lim = p.M - m0 - (odd ? 1 : 0);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t mine = pack2<kDtype>(v[2 * j] * al, v[2 * j + 1] * al);
            const uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
            const uint32_t w = odd ? prmt(other, mine, 0x7632) : prmt(mine, other, 0x5410);
            if (2 * j < lim) {
                uint16_t* d = o + static_cast<int64_t>(2 * j) * p.ldc;
                if (vec) {
                    *reinterpret_cast<uint32_t*>(d) = w;
                } else {
                    d[0] = static_cast<uint16_t>(w);
                    d[1] = static_cast<uint16_t>(w >> 16);
                }
            }
        }
    }
}

template <bool kTma, int kDtype, bool kNMajor>
__global__ void __launch_bounds__(kThreadsL, 1)
gemm_large_kernel(const __grid_constant__ LargeParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    __shared__ __align__(8) uint64_t bars[2 * kMaxStagesL + 4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bn = p.bn, stages = p.stages, nch = p.nch;
    const uint32_t b_codes = static_cast<uint32_t>(bn) * 128u;
    const uint32_t stage_bytes = kABytes + b_codes + static_cast<uint32_t>(nch) * 2048u;
    const uint32_t bar_full = smem_u32(&bars[0]), bar_empty = smem_u32(&bars[kMaxStagesL]);
    const uint32_t bar_accfull = smem_u32(&bars[2 * kMaxStagesL]), bar_accempty = bar_accfull + 16;
    const int n_acc = bn <= 128 ? 2 : 1;             // accumulator buffers in 256 columns

    if (warp == 0 && lane < 2 * kMaxStagesL + 4) {
        mbar_init(bar_full + 8 * lane, lane >= 2 * kMaxStagesL + 2 ? kEpiWarps : 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(smem_u32(&s_tmem), kTmemColsL);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();

    WaitFail wf;
    if (warp == 0) {
        // ---------------- producer (the whole warp walks, one elected lane issues) ------------
        const bool lead = elect_one();
        // tokens are read by every column of tiles, a weight tile by tiles_m CTAs at about the same time
        const uint64_t keep = l2_policy_evict_last();
        const uint64_t policy = p.tiles_m > 1 ? l2_policy_evict_normal() : l2_policy_evict_first();
        auto load_a = [&](const Segment& sg, int kb, int s) {
            const int nt = sg.tile / p.tiles_m;
            const uint32_t dst = ring + s * stage_bytes;
            if (kTma) {
                tma_load_2d(dst, &p.map_w, kb * 128, nt * kRows, bar_full + 8 * s, policy);
                bulk_g2s(dst + kACodes, p.wsf + (static_cast<int64_t>(nt) * p.k64 + kb * 4) * 512, 2048, bar_full + 8 * s, policy);
            } else {
                bulk_g2s(dst, p.w + (static_cast<int64_t>(nt) * p.kblocks + kb) * kABytes, kABytes, bar_full + 8 * s, policy);
            }
        };
        auto load_b = [&](const Segment& sg, int kb, int s, int valid_ch) {
            const int mt = sg.tile % p.tiles_m;
            const uint32_t dst = ring + s * stage_bytes + kABytes;
            if (kTma) {
                tma_load_2d(dst, &p.map_x, kb * 128, mt * bn, bar_full + 8 * s, keep);
                for (int j = 0; j < valid_ch; ++j)
                    bulk_g2s(dst + b_codes + j * 2048, p.xsf + (static_cast<int64_t>(mt * nch + j) * p.k64 + kb * 4) * 512,
                             2048, bar_full + 8 * s, keep);
            } else {
                const uint32_t bytes = b_codes + static_cast<uint32_t>(nch) * 2048u;
                bulk_g2s(dst, p.x + (static_cast<int64_t>(mt) * p.kblocks + kb) * bytes, bytes, bar_full + 8 * s, keep);
            }
        };
        auto chunks_of = [&](const Segment& sg) {     // 128-row scale chunks of the tile that exist in xsf
            if (!kTma) return nch;
            const int rows = p.M - (sg.tile % p.tiles_m) * bn;
            return min(nch, (rows + 127) >> 7);
        };
        // The weight does not depend on the kernel before: the weight half of the first stages is
        // requested ahead of the wait, the token half behind it.
        Walker wa(p);
        Segment sa;
        int pre = 0;
        {
            bool more = wa.next(p, sa);
            int kb = more ? sa.k0 : 0;
            while (more && pre < stages) {
                if (lead) {
                    mbar_expect_tx(bar_full + 8 * pre, kABytes + b_codes + static_cast<uint32_t>(chunks_of(sa)) * 2048u);
                    load_a(sa, kb, pre);
                }
                ++pre;
                if (++kb == sa.k1) { more = wa.next(p, sa); kb = sa.k0; }
            }
        }
        pdl_wait_prior();
        Walker wk(p);
        Segment sg;
        int i = 0;
        uint32_t s = 0, phase = 1;                    // phase the empty barrier must have completed
        while (!wf.failed && wk.next(p, sg)) {
            const int ch = chunks_of(sg);
            for (int kb = sg.k0; kb < sg.k1; ++kb, ++i) {
                if (i >= stages && !wf.wait(bar_empty + 8 * s, phase)) break;
                if (lead) {
                    if (i >= pre) {
                        mbar_expect_tx(bar_full + 8 * s, kABytes + b_codes + static_cast<uint32_t>(ch) * 2048u);
                        load_a(sg, kb, s);
                    }
                    load_b(sg, kb, s, ch);
                }
                __syncwarp();
                if (++s == static_cast<uint32_t>(stages)) { s = 0; phase ^= 1u; }
            }
        }
        if (wf.failed)                                 // let the copies in flight land before the CTA goes
            for (int j = max(0, i - stages); j < i; ++j) mbar_wait_bounded(bar_full + 8 * (j % stages), (j / stages) & 1, 100000u);
    } else if (warp == 1) {
        // ---------------- MMA issuer -----------------------------------------------------------
        const bool lead = elect_one();
        const uint32_t idesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(bn >> 3) << 17) | (1u << 27);
        Walker wk(p);
        Segment sg;
        uint32_t s = 0, phase = 0;
        int i = 0;
        for (int t = 0; !wf.failed && wk.next(p, sg); ++t) {
            const int buf = n_acc == 2 ? (t & 1) : 0;
            const int use = n_acc == 2 ? (t >> 1) : t;           // how often this buffer was used before
            if (use > 0 && !wf.wait(bar_accempty + 8 * buf, (use - 1) & 1)) break;
            tc_fence_after();
            const uint32_t d = tmem + buf * 128;
            for (int kb = sg.k0; kb < sg.k1; ++kb, ++i) {
                if (!wf.wait(bar_full + 8 * s, phase)) break;
                tc_fence_after();
                const uint32_t a_smem = ring + s * stage_bytes;
                const uint64_t a_desc = desc_operand(a_smem), b_desc = desc_operand(a_smem + kABytes);
                const uint64_t sa_desc = desc_scales(a_smem + kACodes), sb_desc = desc_scales(a_smem + kABytes + b_codes);
                const uint32_t sfa = tmem + kColSfaL + (i & 1) * 16, sfb = tmem + kColSfbL + (i & 1) * 32;
                if (lead) {
                    const uint32_t more = kb > sg.k0 ? 1u : 0u;
                    if (p.k64 - kb * 4 < 4) {                     // K % 256 == 128: the last block has two of four
                        for (int k = 0; k < 2; ++k) {
                            tc_cp_scales(sfa + 4 * k, sa_desc + 32 * k);
                            for (int j = 0; j < nch; ++j) tc_cp_scales(sfb + 4 * nch * k + 4 * j, sb_desc + 128 * j + 32 * k);
                        }
                        for (int k = 0; k < 2; ++k)
                            tc_mma_nvf4(d, a_desc + 2 * k, b_desc + 2 * k, idesc, sfa + 4 * k, sfb + 4 * nch * k, k == 0 ? more : 1u);
                    } else if (nch == 1) {
                        issue_block<1>(d, a_desc, b_desc, sa_desc, sb_desc, idesc, sfa, sfb, more);
                    } else {
                        issue_block<2>(d, a_desc, b_desc, sa_desc, sb_desc, idesc, sfa, sfb, more);
                    }
                    tc_commit(bar_empty + 8 * s);
                }
                __syncwarp();
                if (++s == static_cast<uint32_t>(stages)) { s = 0; phase ^= 1u; }
            }
            if (lead) tc_commit(bar_accfull + 8 * buf);
            __syncwarp();
        }
    } else {
        // ---------------- epilogue (warps 2..9) ------------------------------------------------
        pdl_wait_prior();                              // out, partials and tickets may still be in use before it
        const int q = warp & 3, half = (warp - 2) >> 2;
        const int row = q * 32 + lane;
        const int cols_half = (((bn >> 4) + 1) >> 1) << 4;
        const int c_lo = half ? cols_half : 0, c_n = half ? bn - cols_half : cols_half;
        const bool vec = kNMajor ? (p.ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0)
                                 : (reinterpret_cast<uintptr_t>(p.out) & 3) == 0;
        Walker wk(p);
        Segment sg;
        for (int t = 0; wk.next(p, sg); ++t) {
            const int buf = n_acc == 2 ? (t & 1) : 0;
            const int use = n_acc == 2 ? (t >> 1) : t;
            const int nt = sg.tile / p.tiles_m, mt = sg.tile - nt * p.tiles_m;
            const int n = nt * kRows + row, m0 = mt * bn;
            wf.wait(bar_accfull + 8 * buf, use & 1);   // after a time-out: walk on, the warps meet at barriers below
            tc_fence_after();
            const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16) + buf * 128 + c_lo;
            const bool shared_tile = sg.k1 - sg.k0 != p.kblocks;
            // drain the whole half into registers, then let the next tile's MMAs at the accumulator
            float v[8][16];
#pragma unroll
            for (int g = 0; g < 8; ++g)
                if (16 * g < c_n) tmem_ld16(taddr + 16 * g, v[g]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_accempty + 8 * buf);
            if (!shared_tile) {
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    if (16 * g < c_n) store16<kDtype, kNMajor>(p, n, m0 + c_lo + 16 * g, v[g], lane, vec);
                continue;
            }
            // stream-K: leave the partial sums, the last CTA of the tile to arrive adds all of them
            const int base = (sg.tile - p.sk_base) * p.kblocks;
            const int first = sk_owner(p, base), last = sk_owner(p, base + p.kblocks - 1);
            auto slot = [&](int c) {                   // CTA c's partial tile: its first or its last segment
                return reinterpret_cast<float4*>(p.partials) +
                       ((2 * static_cast<int64_t>(c) + (sk_start(p, c) >= base ? 0 : 1)) * bn + c_lo) / 4 * kRows + row;
            };
            {
                float4* mine = slot(blockIdx.x);
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    if (16 * g < c_n) {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            __stcg(mine + (4 * g + j) * kRows, make_float4(v[g][4 * j], v[g][4 * j + 1], v[g][4 * j + 2], v[g][4 * j + 3]));
                    }
            }
            named_barrier(1, kEpiWarps * 32);
            if (tid == 64) {
                __threadfence();
                const unsigned got = atomicAdd(p.tickets + sg.tile - p.sk_base, 1u);
                s_last = got == static_cast<unsigned>(last - first) ? 1 : 0;
                if (s_last) p.tickets[sg.tile - p.sk_base] = 0u;
                __threadfence();
            }
            named_barrier(1, kEpiWarps * 32);
            if (s_last) {
                // two parts: the sum of two does not depend on their order, so this CTA's stays in registers;
                // more: all are added in K order, this CTA's own read back like the others
                const bool two = last - first == 1;
#pragma unroll 1
                for (int c = first; c <= last; ++c) {
                    if (two && c == static_cast<int>(blockIdx.x)) continue;
                    const float4* src = slot(c);
                    const bool add = two || c != first;
#pragma unroll
                    for (int g = 0; g < 8; ++g)
                        if (16 * g < c_n) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float4 t = __ldcg(src + (4 * g + j) * kRows);
                                v[g][4 * j] = add ? v[g][4 * j] + t.x : t.x;
                                v[g][4 * j + 1] = add ? v[g][4 * j + 1] + t.y : t.y;
                                v[g][4 * j + 2] = add ? v[g][4 * j + 2] + t.z : t.z;
                                v[g][4 * j + 3] = add ? v[g][4 * j + 3] + t.w : t.w;
                            }
                        }
                }
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    if (16 * g < c_n) store16<kDtype, kNMajor>(p, n, m0 + c_lo + 16 * g, v[g], lane, vec);
            }
            named_barrier(1, kEpiWarps * 32);          // s_last is written again for the next shared tile
        }
    }

    if (wf.failed && lane == 0) report_timeout(&g_large_status, 6);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemColsL);
    }
}

// ---- host side ---------------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeFn>(sym);
    });
    return fn;
}

// [rows, K/2] bytes, box of 128 bytes x box_rows, 128-byte swizzle; rows past the end read as zero.
bool code_map(const void* p, int rows, int K, int box_rows, CUtensorMap* out) {
    EncodeFn fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K / 2), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K / 2)};
    const cuuint32_t box[2] = {128, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(p), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct LargePlan {
    int bn, nch, tiles_m, tiles, kblocks, stages, grid;
    int dp_rounds, sk_base, sk_ctas;
    size_t smem, token_bytes, ticket_bytes, partial_bytes;
};

int g_large_bn = 0, g_large_sk = -1, g_large_min_m = 0;

// Tile width and schedule by an estimate of the time in nanoseconds, for G SMs.
bool make_large_plan(int M, int N, int K, bool row_major, int G, LargePlan* plan) {
    const int kblocks = (K + kBK - 1) / kBK, tiles_n = N / kRows;
    double best = 1e30;
    bool found = false;
    const int mt0 = (M + 255) / 256;
    for (int mt = mt0; mt <= mt0 + 4; ++mt) {
        int bn = ((M + mt - 1) / mt + 15) / 16 * 16;
        if (g_large_bn) bn = g_large_bn;
        if (row_major && M > bn) bn = (bn + 127) / 128 * 128;     // a tile starts at a scale chunk
        if (bn > 256) continue;
        const int tiles_m = (M + bn - 1) / bn;
        const int64_t tiles = static_cast<int64_t>(tiles_m) * tiles_n;
        if (tiles * kblocks > 0x3fffffff) continue;
        const int nch = (bn + 127) / 128;
        const double stage = kStageBase + kStagePerToken * bn, epi = bn > 128 ? 500.0 : 100.0;
        const int full = static_cast<int>(tiles / G);
        auto consider = [&](int dp, int ctas, double t) {
            if (t >= best) return;
            best = t;
            found = true;
            plan->bn = bn; plan->nch = nch; plan->tiles_m = tiles_m; plan->tiles = static_cast<int>(tiles);
            plan->kblocks = kblocks; plan->dp_rounds = dp; plan->sk_ctas = ctas;
        };
        if (g_large_sk != 1) {
            const int rounds = static_cast<int>((tiles + G - 1) / G);
            consider(rounds, 0, rounds * (kblocks * stage + epi));
        }
        if (g_large_sk == 0) continue;
        for (int dp = full; dp >= 0 && dp >= full - 1; --dp) {
            const int64_t rest = tiles - static_cast<int64_t>(dp) * G;
            if (rest <= 0) continue;
            for (int parts = 2; parts <= 9; ++parts) {             // 9: every CTA
                const int64_t want = rest * parts;
                const int ctas = parts == 9 || want > G ? G : static_cast<int>(want);
                if (rest * kblocks < ctas) continue;
                const double share = static_cast<double>(rest) / ctas;                // tiles per CTA
                const double gather = static_cast<double>(ctas) / rest + 1.0;         // parts of a shared tile, about
                consider(dp, ctas, dp * (kblocks * stage + epi) + (share * kblocks + 1.0) * stage + epi + kFixBase +
                                       gather * kFixPerPart * ((bn + 63) / 64));
                if (ctas == G) break;
            }
        }
    }
    if (!found) return false;
    const size_t stage_bytes = kABytes + plan->bn * 128 + plan->nch * 2048;
    int stages = static_cast<int>((kSmemBudget - 1024) / stage_bytes);
    plan->stages = stages > kMaxStagesL ? kMaxStagesL : stages;
    plan->smem = plan->stages * stage_bytes + 1024;
    plan->grid = plan->dp_rounds > 0 && plan->tiles >= G ? G : (plan->dp_rounds > 0 ? plan->tiles : plan->sk_ctas);
    plan->sk_base = plan->sk_ctas > 0 ? plan->dp_rounds * G : plan->tiles;
    plan->token_bytes = (static_cast<size_t>(plan->tiles_m) * kblocks * (plan->bn * 128 + plan->nch * 2048) + 255) / 256 * 256;
    plan->ticket_bytes = plan->sk_ctas ? (static_cast<size_t>(plan->tiles - plan->sk_base) * 4 + 255) / 256 * 256 : 0;
    plan->partial_bytes = static_cast<size_t>(2) * plan->sk_ctas * plan->bn * kRows * 4;
    return true;
}

// A call asks three times (scratch size, its check, launch) and plans once: 0.3 us each.
bool plan_large(int M, int N, int K, bool row_major, LargePlan* plan) {
    struct Last { int M, N, K, G, bn, sk; bool row_major, found; LargePlan plan; };
    static thread_local Last last = {};
    const int G = device_sm_count();
    if (last.M != M || last.N != N || last.K != K || last.G != G || last.bn != g_large_bn || last.sk != g_large_sk ||
        last.row_major != row_major) {
        last = Last{M, N, K, G, g_large_bn, g_large_sk, row_major, false, {}};
        last.found = make_large_plan(M, N, K, row_major, G, &last.plan);
    }
    *plan = last.plan;
    return last.found;
}

using Kern = void (*)(LargeParams);

constexpr int kInstances = 9;

cudaError_t launch_with_pdl(int instance, const LargePlan& plan, const LargeParams& p, cudaStream_t stream) {
    // packed operands, then row-major ones with M-major and with N-major output; bf16, fp16, fp32
    static const Kern table[kInstances] = {
        gemm_large_kernel<false, 0, false>, gemm_large_kernel<false, 1, false>, gemm_large_kernel<false, 2, false>,
        gemm_large_kernel<true, 0, false>, gemm_large_kernel<true, 1, false>, gemm_large_kernel<true, 2, false>,
        gemm_large_kernel<true, 0, true>, gemm_large_kernel<true, 1, true>, gemm_large_kernel<true, 2, true>};
    const Kern kern = table[instance];
    static std::atomic<bool> attr_done[kInstances][64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_done[instance][dev].load(std::memory_order_relaxed)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[instance][dev].store(true, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(plan.grid));
    cfg.blockDim = dim3(kThreadsL);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gemv_tuning().use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

template <typename... Params, typename... Args>
cudaError_t launch_small(void (*kern)(Params...), dim3 grid, int threads, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gemv_tuning().use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<Params>(args)...);
}

void fill_common(const LargePlan& plan, LargeParams* p, void* out, int M, int N, int K, float alpha, bool n_major) {
    p->out = out;
    p->ldc = n_major ? M : N;
    p->M = M; p->N = N;
    p->bn = plan.bn; p->nch = plan.nch; p->tiles = plan.tiles; p->tiles_m = plan.tiles_m;
    p->kblocks = plan.kblocks; p->k64 = K / 64; p->stages = plan.stages;
    p->dp_rounds = plan.dp_rounds; p->sk_base = plan.sk_base; p->sk_ctas = plan.sk_ctas;
    if (plan.sk_ctas > 0) {
        const int total = (plan.tiles - plan.sk_base) * plan.kblocks;
        p->sk_q = total / plan.sk_ctas;
        p->sk_r = total % plan.sk_ctas;
    }
    p->alpha = alpha;
}

}  // namespace

// Tokens from which the row-major operands of the raw gemm operator take this path.
constexpr int kLargeMinM = 33;

// Tokens from which the packed linear takes it, where the caller can give it scratch: the device's side of the
// choice. Up to 16 tokens the decode kernel makes one pass over the weight as well and needs no second launch; its
// CTAs each quantize the tokens of their K part, which grows with the tokens, while this path pays a few us for
// partial sums where the weight has few row tiles and long rows. Measured in CUDA graphs, us, decode kernel / this one:
//   N >= 6 K       34816x5120: 13 tokens 25.6 / 21.3, 16 tokens 26.4 / 21.5; 12288x2048: 13 tokens 8.2 / 6.4;
//                  but (N >= 16 K) 24576x1024: 13 tokens 6.1 / 6.8, 17 tokens 8.1 / 6.9
//   N >= 1.5 K     12288x4096: 17 tokens 15.3 / 10.5; 10240x5120: 17 tokens 15.9 / 11.6; 6144x4096: 17 tokens 10.0 / 9.7
//   N >= K         4096x4096: 25 tokens 9.9 / 9.4, 32 tokens 11.3 / 9.5
//   below          4096x12288: 24 tokens 13.2 / 15.7, 32 tokens 15.7 / 15.7; 1280x5120: 32 tokens 9.6 / 11.2
int large_min_m(int N, int K) {
    const int64_t n = N, k = K;
    return n >= 6 * k && n < 16 * k ? 13 : 2 * n >= 3 * k ? 17 : n >= k ? 25 : kLargeMinM;
}

// What the entry point takes.
bool large_accepts(int M, int N, int K) {
    return N > 0 && K > 0 && N % kRows == 0 && K % 128 == 0 && M >= (g_large_min_m ? g_large_min_m : large_min_m(N, K));
}

bool large_pays(int M, int N, int K) {
    if (!large_accepts(M, N, K)) return false;
    if (g_large_min_m) return true;
    const int G = device_sm_count(), tiles = N / kRows, kblocks = (K + kBK - 1) / kBK;
    // A narrow weight with rows of 31 or 32 K blocks: the longest that still run as whole tiles here (0.48 us a
    // block), while two launches of the decode kernel give each CTA one block and one token to add up. 33 / 48 / 64
    // tokens: 640x8192 13.0 / 14.0 / 14.3, here 15.5 / 15.7 / 15.9; 1280x8192 14.3 / 15.5 / 18.6, here 16.0 / 15.9 / 16.2;
    // 30 blocks, 1024x7680: 14.9 / 16.0 / 17.4, here 14.8 / 14.8 / 15.0; 33, 1792x8320: 17.2 / 18.4 / 22.4, here 16.8.
    if (M <= 64 && kblocks > 30 && kblocks <= 32 && tiles <= (M <= 48 ? 16 : 8)) return false;
    // Up to 16 tokens both kernels are bound by the weight, and here 1 to 1.5 tiles per SM cost two full rounds of
    // 0.48 us a K block. 20480x2048: 13 tokens 8.9 / 10.7, 16 tokens 9.8 / 10.8; 24576x4096: 16 tokens 17.4 / 18.5;
    // but 24064x2304, where the decode kernel splits K: 16 tokens 15.3 / 11.5; 22528x3072: 16 tokens 16.4 / 15.1.
    if (M <= 16 && tiles > G && 2 * tiles < 3 * G) return packed_time_us(M, N, K) > 3.9 + 0.96 * kblocks;
    return true;
}

size_t large_scratch_bytes(int M, int N, int K) {
    LargePlan plan;
    if (!large_accepts(M, N, K) || !plan_large(M, N, K, false, &plan)) return 0;
    return plan.token_bytes + plan.ticket_bytes + plan.partial_bytes;
}

// The host's side: a second launch and the scratch bring a call to 12 us or more even where the device needs 5, while
// a call of the decode kernel ends at 8.5. So up to 32 tokens (one launch of it) that kernel keeps what it does in
// less. Measured, us a call: 6144x1024, 16 tokens 8.5 / 12.0; 12288x2048, 16 tokens 8.9 / 12.0; 4096x4096, 32 tokens
// 11.4 / 12.2; 6144x2048, 32 tokens 13.1 / 12.2; 8192x3072, 20 tokens 13.0 / 12.1.
constexpr double kLargeCallUs = 12.0;

int large_route(int M, int N, int K) {
    if (!large_pays(M, N, K)) return NVFP4R_ROUTE_PACKED;
    return g_large_min_m || M > 32 || packed_time_us(M, N, K) >= kLargeCallUs ? NVFP4R_ROUTE_SCRATCH : NVFP4R_ROUTE_SCRATCH_CAPTURED;
}

cudaError_t launch_linear_large(const PackedLinearArgs& g, void* scratch, cudaStream_t stream) {
    LargePlan plan;
    if (!plan_large(g.M, g.N, g.K, false, &plan)) return cudaErrorInvalidConfiguration;
    uint8_t* tokens = static_cast<uint8_t*>(scratch);
    LargeParams p = {};
    fill_common(plan, &p, g.out, g.M, g.N, g.K, g.alpha, false);
    p.w = static_cast<const uint8_t*>(g.packed);
    p.x = tokens;
    p.tickets = reinterpret_cast<unsigned*>(tokens + plan.token_bytes);
    p.partials = reinterpret_cast<float*>(tokens + plan.token_bytes + plan.ticket_bytes);
    const dim3 qgrid(static_cast<unsigned>(g.M), static_cast<unsigned>((g.K / kBlockElems + 255) / 256));
    cudaError_t e = launch_small(quant_pack_kernel, qgrid, 256, stream, static_cast<const __nv_bfloat16*>(g.xb), g.xb_stride,
                                 g.K, g.gs, g.rcp_mode == kRcpExact, tokens, plan.bn, plan.nch, plan.kblocks,
                                 p.tickets, plan.tiles - plan.sk_base);
    if (e != cudaSuccess) return e;
    return launch_with_pdl(g.out_dtype, plan, p, stream);
}

// The raw operator on row-major operands. *taken stays false (nothing launched) where the workspace
// does not hold what this path needs or a tensor map cannot be made: the caller's other kernel runs.
cudaError_t launch_gemm_large(const TcLinearArgs& g, cudaStream_t stream, bool* taken) {
    *taken = false;
    LargePlan plan;
    if (g.xb != nullptr || g.M < (g_large_min_m ? g_large_min_m : kLargeMinM) || !plan_large(g.M, g.N, g.K, true, &plan))
        return cudaSuccess;
    LargeParams p = {};
    fill_common(plan, &p, g.out, g.M, g.N, g.K, g.alpha, g.c_n_major);
    if (!code_map(g.w, g.N, g.K, kRows, &p.map_w) || !code_map(g.a_codes, g.M, g.K, plan.bn, &p.map_x)) return cudaSuccess;
    p.wsf = static_cast<const uint8_t*>(g.wsf_swizzled);
    p.xsf = static_cast<const uint8_t*>(g.a_sf_swizzled);
    // The workspace, tickets included, is shared with the decode-sized kernel: both leave the tickets zero.
    GemmScratch scratch = {};
    cudaError_t e = cudaSuccess;
    if (plan.sk_ctas > 0 && !gemm_scratch(g.workspace, g.workspace_bytes, plan.ticket_bytes, plan.partial_bytes, stream,
                                          &scratch, &e))
        return cudaSuccess;
    if (e != cudaSuccess) return e;
    p.tickets = scratch.tickets;
    p.partials = scratch.partials;
    *taken = true;
    e = launch_with_pdl((g.c_n_major ? 6 : 3) + g.out_dtype, plan, p, stream);
    return e == cudaSuccess ? gemm_scratch_done(scratch, stream) : e;
}

void set_large_tuning(int min_m, int bn, int stream_k) {
    g_large_min_m = min_m;
    g_large_bn = bn;
    g_large_sk = stream_k;
}

cudaError_t set_status_mirror_large(int* p) { return set_status_mirror_here(p); }

cudaError_t read_and_clear_large_status(int* flag) {
    cudaError_t e = cudaMemcpyFromSymbol(flag, g_large_status, sizeof(int));
    if (e != cudaSuccess) return e;
    const int zero = 0;
    return cudaMemcpyToSymbol(g_large_status, &zero, sizeof(int));
}

}  // namespace nvfp4r
