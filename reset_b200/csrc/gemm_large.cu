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
//              A pipeline stage (256 K-elements) is two 1-D bulk copies, in a CTA of a pair
//              three tensor-map loads of the same bytes (weight, its half of the codes, token scales).
//   row-major  codes through 2-D tensor maps (128-byte swizzle), scales in the 128x4-tiled layout as
//              512-byte chunks: the operands of the raw gemm operator.
//
// CTAs of ten warps, one per SM: warp 0 producer, warp 1 MMA issuer, warps 2-9 epilogue (two
// per TMEM lane quadrant, each half of the columns). Four schedules, chosen by an estimate of the time:
//   whole tiles  CTA c computes tiles c, c + G, ...
//   stream-K     after the rounds of whole tiles the K blocks of the tiles that are left, laid end to end, are cut into
//                one equal range for each of `sk_ctas` CTAs. A tile that two or more CTAs share is summed from fp32
//                partials in scratch, in K order, by the one that finishes last (atomic ticket; nothing waits, results
//                do not depend on the order of arrival).
//   cluster      a cluster of `split` CTAs takes one tile, each CTA an equal share of the K blocks. Each sends its partial
//                sums of the columns that a peer owns into that peer's shared memory (the ring, idle by then), and
//                every CTA adds up and stores its own columns, in K order. The hardware places a cluster as a whole,
//                so nothing waits for a CTA that might not be running, and no scratch is needed.
//   pairs        two SMs on one tile of 256 weight rows (cta_group::2): each holds its 128 rows and half of the tokens,
//                38 KB a stage instead of 55 KB at 256 tokens; one of the two issues for both, and the other's loads
//                complete on its barriers. For many tokens, where the bytes are the time.
//
// What bounds it. Few tiles: the chain launch - quantizer - launch - first stage - MMAs - stores, of which a K block is
// 0.24 us: 515 clocks of the issuing warp (12 tcgen05 instructions at 17 to 25 clocks, a wait, a commit) against 218 for
// the tensor pipe at 16 tokens. Many tokens: the bytes that the SMs take in from L2, 13 to 15 TB/s over all of them; MMAs
// alone would run at 107 bytes a clock and SM without pairing, 74 with, and the loads get 55 to 60.
// The producer's addresses are worked out once per segment and it was 740 clocks a stage before, more than the issuer;
// the issuer is straight-line code per K block (rolled loops made each tcgen05 instruction wait for its operands).
// Device time in a CUDA graph, weights cold, us, one CTA a tile or stream-K with all of that before -> after:
//   10240x5120  45 tokens 12.4 -> 10.1     6144x4096  333 tokens 13.9 -> 11.2     34816x5120  16 tokens 21.9 -> 19.9
//   1024x4096   16 tokens 8.5 -> 6.1 (clusters of 4)    4096x12288 128 tokens, quant + gemm 21.3 -> 14.0 (clusters of 4)
//   24576x4096  512 tokens 32.5 -> 28.7, 1300 69.4 -> 57.0, 2048 104.9 -> 85 to 88 (pairs)
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

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
constexpr int kStoreChunk = 32 * kRows * 2;          // 32 tokens x 128 rows of a 16-bit output on their way to memory
constexpr int kStoreBytes = 2 * kStoreChunk;         // one for each column half
constexpr int kSmemBudget = 225 * 1024;              // dynamic part, 1 KB of it for alignment
constexpr int kMapRow = 1024;                        // contiguous operands of a pair as a map: bytes of a row
constexpr int kPairTuning = 9;                       // set_large_tuning: pairs of SMs
constexpr int kMaxSplit = 8;                         // the largest cluster that every device can place
// Time model of plan_large, nanoseconds, fitted to sweeps over tile widths and schedules (eight weights, 16 .. 700
// tokens). A K block costs the issuing warp 235 + 0.17 per token of the tile (30 more for the second chunk of token
// scales), unless the SMs at work take in more than 15.5 TB/s from L2 together or the weight more than 6.3 TB/s from
// memory. The last tile's stores take 10.5 per token, those of a tile before it 6,
// beside the next tile's MMAs; where the accumulators overlap these wait 300.
// A shared stream-K tile: partial stores, fence and ticket, then a trip to L2 per part and 32 columns. A cluster: two
// cluster barriers, each CTA's partial sums sent to the peers and read back.
constexpr double kStageBase = 235.0, kStagePerToken = 0.17, kStageChunk = 30.0, kL2Rate = 15500.0, kHbmRate = 6300.0;
constexpr double kStorePerToken = 10.5, kStoreWarm = 6.0, kStoreWait = 300.0, kFixBase = 2000.0, kFixPerPart = 400.0;
constexpr double kSplitBase = 1100.0, kSplitPerToken = 12.0, kSplitPerPartToken = 2.2, kSecondWave = 3500.0;
constexpr double kPairFix = 500.0;
constexpr uint32_t kTmemColsL = 512;
// Tensor memory, 512 columns: two accumulators and the scales of a K block (16 + 32 columns; twice that, so that the next
// block's copies pass the MMAs of this one, where the accumulators leave room). Two accumulators of more than 232 tokens
// overlap: the tokens that both hold are stored first, then the next tile's MMAs may begin.
constexpr int kTwoScales = 208, kNoOverlap = 232;
__host__ __device__ constexpr int acc_stride(int bn) { return bn <= kTwoScales ? kTwoScales : bn <= kNoOverlap ? kNoOverlap : 2 * kNoOverlap - bn; }
__host__ __device__ constexpr int acc_overlap(int bn) { return bn > kNoOverlap ? 2 * (bn - kNoOverlap) : 0; }
constexpr uint32_t kColSfaL = 416, kColSfbL = 448, kColSfa1 = 464, kColSfb1 = 480;

struct alignas(64) LargeParams {
    CUtensorMap map_w, map_x;                        // row-major form: codes; packed form, pairs: weight blocks, token codes
    const uint8_t* w;                                // packed weight blocks
    const uint8_t* x;                                // packed token blocks
    const uint8_t* wsf;                              // row-major form: 128x4-tiled scales
    const uint8_t* xsf;
    void* out;
    int64_t ldc;
    int M, N, bn, nch, tiles, tiles_m, kblocks, k64; // nch = 128-row scale chunks per token tile
    int stages;
    int split, split_cols;                           // cluster schedule: CTAs per tile (else 1), columns that each sums up
    int dp_rounds, sk_base, sk_ctas, sk_q, sk_r;     // stream-K from tile sk_base on: sk_q (+1 for the first sk_r) K blocks per CTA
    float alpha;
    float* partials;                                 // [2 * sk_ctas][bn / 4][128][4]
    unsigned* tickets;                               // [tiles], zero before the launch, left zero
};

struct alignas(64) PairParams : LargeParams {
    CUtensorMap map_xsf, map_wsf;                    // token scales; row-major form: weight scales
};
template <bool kPair> using ParamsOf = std::conditional_t<kPair, PairParams, LargeParams>;

__device__ int g_large_status = 0;

// ---- token quantizer -------------------------------------------------------------------------
// One thread per 16-element block and row, kR rows a CTA with their loads in flight together; four lanes share one
// 32-bit store of scales. Also clears the tickets of the GEMM that follows.
template <int kR>
__global__ void __launch_bounds__(256)
quant_pack_kernel(const __nv_bfloat16* __restrict__ x, int64_t x_row_stride, int M, int K, const float* __restrict__ gs_ptr,
                  bool exact, uint8_t* __restrict__ packed, int bn, int nch, int kblocks,
                  unsigned* __restrict__ tickets, int n_tickets) {
    pdl_launch_dependents();
    const int row0 = blockIdx.x * kR;
    int mt = row0 / bn, r = row0 - mt * bn;
    const int col = blockIdx.y * 256 + threadIdx.x;
    const float gs = __ldg(gs_ptr);
    const QuantScales q = exact ? make_quant_scales<kRcpExact>(gs) : make_quant_scales<kRcpApprox>(gs);
    pdl_wait_prior();
    if (blockIdx.y == 0)
        for (int i = blockIdx.x * 256 + threadIdx.x; i < n_tickets; i += gridDim.x * 256) tickets[i] = 0u;
    if (col >= K / kBlockElems) return;               // K % 128 == 0: groups of eight lanes leave together
    uint4 lo[kR], hi[kR];
#pragma unroll
    for (int i = 0; i < kR; ++i) {
        const int row = min(row0 + i, M - 1);
        const uint4* src = reinterpret_cast<const uint4*>(x + row * x_row_stride + static_cast<int64_t>(col) * kBlockElems);
        lo[i] = __ldg(src);
        hi[i] = __ldg(src + 1);
    }
    const int kb = col >> 4, b = col & 15;
    const unsigned live = __activemask();
    const int tile_bytes = bn * 128 + nch * 2048;
    uint8_t* base = packed + (static_cast<int64_t>(mt) * kblocks + kb) * tile_bytes;
#pragma unroll
    for (int i = 0; i < kR; ++i) {
        if (row0 + i >= M) break;
        uint32_t c[2];
        const uint32_t sf = quantize_block16_rt(lo[i], hi[i], q, exact, c);
        *reinterpret_cast<uint2*>(base + swz128(r, b * 8)) = make_uint2(c[0], c[1]);
        uint32_t s4 = sf << (8 * (b & 3));
        s4 |= __shfl_xor_sync(live, s4, 1);
        s4 |= __shfl_xor_sync(live, s4, 2);
        if ((b & 3) == 0)
            *reinterpret_cast<uint32_t*>(base + bn * 128 + (r >> 7) * 2048 + (b >> 2) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4) = s4;
        if (++r == bn) { r = 0; base += static_cast<int64_t>(kblocks) * tile_bytes; }
    }
}

// ---- work of one CTA -------------------------------------------------------------------------
struct Segment { int tile, k0, k1; };

struct Walker {
    int round = 0, cur, end, unit, units;             // unit: this CTA, or its pair
    __device__ __forceinline__ Walker(const LargeParams& p, bool pair) {
        const int c = blockIdx.x;
        unit = pair ? c >> 1 : c;
        units = pair ? gridDim.x / 2 : gridDim.x;
        cur = c * p.sk_q + min(c, p.sk_r);
        end = c < p.sk_ctas ? cur + p.sk_q + (c < p.sk_r ? 1 : 0) : cur;
    }
    __device__ __forceinline__ bool next(const LargeParams& p, Segment& s) {
        if (p.split > 1) {
            s.tile = static_cast<int>(blockIdx.x) / p.split;
            const int part = static_cast<int>(blockIdx.x) - s.tile * p.split;
            s.k0 = p.kblocks * part / p.split;
            s.k1 = p.kblocks * (part + 1) / p.split;
            return round++ == 0;
        }
        if (round < p.dp_rounds) {
            s.tile = unit + round * units;
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
template <int kChunks, int kSteps, bool kPair>
__device__ __forceinline__ void issue_block(uint32_t d, uint64_t a, uint64_t b, uint64_t sa, uint64_t sb, uint32_t idesc,
                                            uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
    const auto cp = [](uint32_t t, uint64_t desc) {
        if (kPair) tc_cp_scales_pair(t, desc);
        else tc_cp_scales(t, desc);
    };
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
        cp(sfa + 4 * k, sa + 32 * k);
#pragma unroll
        for (int j = 0; j < kChunks; ++j) cp(sfb + 4 * kChunks * k + 4 * j, sb + 128 * j + 32 * k);
    }
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
        if (kPair) tc_mma_nvf4_pair(d, a + 2 * k, b + 2 * k, idesc, sfa + 4 * k, sfb + 4 * kChunks * k, k == 0 ? accumulate : 1u);
        else tc_mma_nvf4(d, a + 2 * k, b + 2 * k, idesc, sfa + 4 * k, sfb + 4 * kChunks * k, k == 0 ? accumulate : 1u);
    }
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

// Stores kCols accumulator columns (tokens m0 .. m0 + kCols - 1) of the tile's 128 rows; the four warps of a column half
// call it together, each lane with its weight row n = n0 + row.
//   N-major         a lane's tokens are contiguous. Where rows are not 16-byte aligned (16-bit output, M % 8 != 0) a warp
//                   turns its 32 rows in shared memory and writes row by row: 32 single stores of a lane each went to 32
//                   rows at once (16384x2048 with 333 tokens 61 us, with 1000 tokens 24).
//   M-major, fp32   the lanes of a warp write 128 contiguous bytes per token.
//   M-major, 16-bit a warp's share of a token is 64 bytes: the half's values meet in shared memory and leave
//                   in 16-byte pieces, 256 contiguous bytes per token. Straight from the registers (pairs of lanes
//                   trading halves, 4 bytes a store) a tile of 128 x 112 took 2.4 us.
struct Store {
    uint8_t* chunk;     // this half's, in shared memory
    int half, row, align;
};

template <int kDtype, bool kNMajor, int kCols>
__device__ __forceinline__ void store_cols(const LargeParams& p, const Store& st, int n0, int m0, float v[kCols]) {
#pragma unroll
    for (int j = 0; j < kCols; ++j) v[j] *= p.alpha;
    if (kNMajor) {
        const int64_t at = static_cast<int64_t>(n0 + st.row) * p.ldc + m0;
        if (kDtype == 2) {
            float* o = static_cast<float*>(p.out) + at;
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                if (m0 + j < p.M) o[j] = v[j];
        } else {
            uint16_t* o = static_cast<uint16_t*>(p.out) + at;
            uint32_t w[kCols / 2];
#pragma unroll
            for (int j = 0; j < kCols / 2; ++j) w[j] = pack2<kDtype>(v[2 * j], v[2 * j + 1]);
            if (st.align == 16 && m0 + kCols <= p.M) {
#pragma unroll
                for (int j = 0; j < kCols / 8; ++j)
                    reinterpret_cast<uint4*>(o)[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
            } else {
                // [row][token pair], 16 words a row, pairs of rows rotated so that neither side meets a bank twice
                const int lane = st.row & 31;
                uint32_t* turn = reinterpret_cast<uint32_t*>(st.chunk) + (st.row - lane) * 16;
#pragma unroll
                for (int j = 0; j < kCols / 2; ++j) turn[lane * 16 + (j ^ (lane >> 1))] = w[j];
                __syncwarp();
                uint16_t* first = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(n0 + st.row - lane) * p.ldc + m0;
                if (st.align >= 4) {                   // M even
                    const int pair = lane & 15;
                    if (pair < kCols / 2 && m0 + 2 * pair < p.M)
#pragma unroll 4
                        for (int i = 0; i < 16; ++i) {
                            const int r = 2 * i + (lane >> 4);
                            *reinterpret_cast<uint32_t*>(first + r * p.ldc + 2 * pair) = turn[r * 16 + (pair ^ i)];
                        }
                } else if (lane < kCols && m0 + lane < p.M) {
#pragma unroll 4
                    for (int r = 0; r < 32; ++r)
                        first[r * p.ldc + lane] = reinterpret_cast<const uint16_t*>(turn + r * 16 + ((lane >> 1) ^ (r >> 1)))[lane & 1];
                }
                __syncwarp();
            }
        }
    } else if (kDtype == 2) {
        float* o = static_cast<float*>(p.out) + static_cast<int64_t>(m0) * p.ldc + n0 + st.row;
        // A test and a product per store cost more than the store: 23680x1024 with 588 tokens 29.2 us, 18.0 without.
        if (m0 + kCols <= p.M) {
#pragma unroll
            for (int j = 0; j < kCols; ++j, o += p.ldc) *o = v[j];
        } else {
#pragma unroll
            for (int j = 0; j < kCols; ++j, o += p.ldc)
                if (m0 + j < p.M) *o = v[j];
        }
    } else {
        uint16_t* mine = reinterpret_cast<uint16_t*>(st.chunk) + st.row;
#pragma unroll
        for (int j = 0; j < kCols / 2; ++j) {
            const uint32_t w = pack2<kDtype>(v[2 * j], v[2 * j + 1]);
            mine[2 * j * kRows] = static_cast<uint16_t>(w);
            mine[(2 * j + 1) * kRows] = static_cast<uint16_t>(w >> 16);
        }
        named_barrier(2 + st.half, kRows);
#pragma unroll
        for (int u = 0; u < kCols / 8; ++u) {
            const int token = u * 8 + (st.row >> 4), piece = st.row & 15;
            if (m0 + token >= p.M) break;
            const uint4 w = *reinterpret_cast<const uint4*>(st.chunk + token * (kRows * 2) + piece * 16);
            uint16_t* o = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(m0 + token) * p.ldc + n0 + piece * 8;
            if (st.align == 16) {
                *reinterpret_cast<uint4*>(o) = w;
            } else {
                const uint32_t e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (st.align == 4) {
                        reinterpret_cast<uint32_t*>(o)[j] = e[j];
                    } else {
                        o[2 * j] = static_cast<uint16_t>(e[j]);
                        o[2 * j + 1] = static_cast<uint16_t>(e[j] >> 16);
                    }
                }
            }
        }
        named_barrier(2 + st.half, kRows);             // read before the next tokens are written
    }
}

// The issuing warp: all lanes walk, one elected lane issues.
template <int kChunks, bool kPair>
__device__ __forceinline__ void issue_all(const LargeParams& p, uint32_t ring, uint32_t tmem, uint32_t bar_full,
                                          uint32_t bar_empty, uint32_t bar_accfull, uint32_t bar_accempty, WaitFail& wf) {
    const bool lead = elect_one();
    const uint32_t b_codes = static_cast<uint32_t>(p.bn) * (kPair ? 64u : 128u);
    const uint32_t stage_bytes = kABytes + b_codes + kChunks * 2048u;
    const uint32_t idesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(p.bn >> 3) << 17) | ((kPair ? 2u : 1u) << 27);
    const int stages = p.stages, stride = acc_stride(p.bn);
    const bool overlap = acc_overlap(p.bn) > 0, two_scales = p.bn <= kTwoScales;
    const auto commit = [](uint32_t bar) {
        if (kPair) tc_commit_pair(bar);
        else tc_commit(bar);
    };
    const int whole = p.k64 >> 2;                     // K % 256 == 128: the last block has two of four steps
    Walker wk(p, kPair);
    Segment sg;
    uint32_t s = 0, phase = 0, odd = 0;
    for (int t = 0; !wf.failed && wk.next(p, sg); ++t) {
        const int buf = t & 1;
        // overlapping accumulators: one barrier, the tile before has left the tokens that both hold; else one per buffer
        const auto emptied = [&](uint32_t bar, uint32_t parity) { return kPair ? wf.wait_cluster(bar, parity) : wf.wait(bar, parity); };
        if (overlap ? t > 0 && !emptied(bar_accempty, (t - 1) & 1) : t > 1 && !emptied(bar_accempty + 8 * buf, ((t >> 1) - 1) & 1)) break;
        tc_fence_after();
        const uint32_t d = tmem + buf * stride;
        uint32_t more = 0;
        for (int kb = sg.k0; kb < sg.k1; ++kb) {
            if (!wf.wait(bar_full + 8 * s, phase)) break;
            tc_fence_after();
            const uint32_t a_smem = ring + s * stage_bytes;
            const uint64_t a_desc = desc_operand(a_smem), b_desc = desc_operand(a_smem + kABytes);
            const uint64_t sa_desc = desc_scales(a_smem + kACodes), sb_desc = desc_scales(a_smem + kABytes + b_codes);
            const uint32_t sfa = tmem + (two_scales ? kColSfaL + odd * 16 : kColSfa1);
            const uint32_t sfb = tmem + (two_scales ? kColSfbL + odd * 32 : kColSfb1);
            if (lead) {
                if (kb < whole) issue_block<kChunks, 4, kPair>(d, a_desc, b_desc, sa_desc, sb_desc, idesc, sfa, sfb, more);
                else issue_block<kChunks, 2, kPair>(d, a_desc, b_desc, sa_desc, sb_desc, idesc, sfa, sfb, more);
                commit(bar_empty + 8 * s);
            }
            __syncwarp();
            more = 1;
            odd ^= 1u;
            if (++s == static_cast<uint32_t>(stages)) { s = 0; phase ^= 1u; }
        }
        if (lead) commit(bar_accfull + 8 * buf);
        __syncwarp();
    }
}

template <bool kTma, int kDtype, bool kNMajor, bool kPair>
__global__ void __launch_bounds__(kThreadsL, 2)
gemm_large_kernel(const __grid_constant__ ParamsOf<kPair> p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    __shared__ __align__(8) uint64_t bars[2 * kMaxStagesL + 4];
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bn = p.bn, stages = p.stages, nch = p.nch;
    const uint32_t b_codes = static_cast<uint32_t>(bn) * (kPair ? 64u : 128u);      // a CTA of a pair holds half of the tokens
    const uint32_t stage_bytes = kABytes + b_codes + static_cast<uint32_t>(nch) * 2048u;
    const int rank = kPair ? static_cast<int>(blockIdx.x & 1) : 0;                  // 0 issues for both
    const uint32_t bar_full = smem_u32(&bars[0]), bar_empty = smem_u32(&bars[kMaxStagesL]);
    const uint32_t bar_accfull = smem_u32(&bars[2 * kMaxStagesL]), bar_accempty = bar_accfull + 16;

    if (warp == 0 && lane < 2 * kMaxStagesL + 4) {
        // a pair: the issuing CTA's accumulators are empty when both are
        const bool acc_empty = lane >= 2 * kMaxStagesL + 2;
        mbar_init(bar_full + 8 * lane, acc_empty ? (kPair ? 2 : 1) * kEpiWarps : 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        if (kPair) tmem_alloc_pair(smem_u32(&s_tmem), kTmemColsL);
        else tmem_alloc(smem_u32(&s_tmem), kTmemColsL);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if (kPair) cluster_sync_all();                     // the peer's barriers exist
    pdl_launch_dependents();

    WaitFail wf;
    if (warp == 0) {
        // ---------------- producer (the whole warp walks, one elected lane issues) ------------
        const bool lead = elect_one();
        // tokens are read by every column of tiles, a weight tile by tiles_m CTAs at about the same time
        const uint64_t keep = l2_policy_evict_last();
        const uint64_t policy = p.tiles_m > 1 ? l2_policy_evict_normal() : l2_policy_evict_first();
        const uint32_t b_bytes = static_cast<uint32_t>(bn) * 128u + static_cast<uint32_t>(nch) * 2048u;      // in memory
        // Where a segment's operands lie, worked out once per segment: with the divisions and products in the block
        // loop a stage cost this warp 740 clocks, more than its MMAs.
        struct Source {
            const uint8_t *a, *b;                     // packed: next block; row-major: next scales
            int ax, ay, by, ch;                       // row-major: code coordinates, scale chunks of the token tile
            int ar, br;                               // pairs: what a and b are, in rows of the maps
        };
        auto source = [&](const Segment& sg) {
            const int t = sg.tile / p.tiles_m, mt = sg.tile - t * p.tiles_m;
            // with an odd number of row tiles the last pair's second CTA repeats the first one's and stores nothing
            const int nt = kPair ? min(2 * t + rank, (p.N / kRows) - 1) : t;
            Source o;
            o.ch = nch;
            if (kTma) {
                o.ax = sg.k0 * 128;
                o.ay = nt * kRows;
                o.by = mt * bn + rank * (bn / 2);
                o.ch = min(nch, (p.M - mt * bn + 127) >> 7);          // chunks that exist in xsf
                const int64_t a = static_cast<int64_t>(nt) * p.k64 + sg.k0 * 4, b = static_cast<int64_t>(mt * nch) * p.k64 + sg.k0 * 4;
                o.a = p.wsf + a * 512;
                o.b = p.xsf + b * 512;
                o.ar = static_cast<int>(a / 2);                       // K % 256 == 0: four chunks a block
                o.br = static_cast<int>(b / 2);
            } else {
                const int64_t a = static_cast<int64_t>(nt) * p.kblocks + sg.k0, b = static_cast<int64_t>(mt) * p.kblocks + sg.k0;
                o.a = p.w + a * kABytes;
                o.b = p.x + b * b_bytes;
                o.ar = static_cast<int>(a) * (kABytes / kMapRow);
                o.br = static_cast<int>(b) * static_cast<int>(b_bytes / kMapRow);
            }
            return o;
        };
        // A pair: all loads of a stage, the peer's too, complete on the issuing CTA's barrier, which expects all of their bytes.
        auto load_a = [&](const Source& o, uint32_t dst, uint32_t bar) {
            const uint32_t bytes = kABytes + b_codes + static_cast<uint32_t>(o.ch) * 2048u;
            if constexpr (kPair) {
                if (rank == 0) mbar_expect_tx(bar, 2 * bytes);
                const uint32_t there = cluster_map(bar, 0);
                if (kTma) {
                    tma_load_2d_pair(dst, &p.map_w, o.ax, o.ay, there, policy);
                    tma_load_2d_pair(dst + kACodes, &p.map_wsf, 0, o.ar, there, policy);
                } else {
                    tma_load_2d_pair(dst, &p.map_w, 0, o.ar, there, policy);
                }
            } else {
                mbar_expect_tx(bar, bytes);
                if (kTma) {
                    tma_load_2d(dst, &p.map_w, o.ax, o.ay, bar, policy);
                    bulk_g2s(dst + kACodes, o.a, 2048, bar, policy);
                } else {
                    bulk_g2s(dst, o.a, kABytes, bar, policy);
                }
            }
        };
        auto load_b = [&](const Source& o, uint32_t dst, uint32_t bar) {
            if constexpr (kPair) {
                const uint32_t there = cluster_map(bar, 0);
                if (kTma) {
                    tma_load_2d_pair(dst, &p.map_x, o.ax, o.by, there, keep);
                    for (int j = 0; j < o.ch; ++j) tma_load_2d_pair(dst + b_codes + j * 2048, &p.map_xsf, 0, o.br + j * (p.k64 / 2), there, keep);
                } else {
                    tma_load_2d_pair(dst, &p.map_x, 0, o.br + rank * static_cast<int>(b_codes / kMapRow), there, keep);
                    tma_load_2d_pair(dst + b_codes, &p.map_xsf, 0, o.br + static_cast<int>(2 * b_codes / kMapRow), there, keep);
                }
            } else if (kTma) {
                tma_load_2d(dst, &p.map_x, o.ax, o.by, bar, keep);
                for (int j = 0; j < o.ch; ++j)
                    bulk_g2s(dst + b_codes + j * 2048, o.b + static_cast<int64_t>(j) * p.k64 * 512, 2048, bar, keep);
            } else {
                bulk_g2s(dst, o.b, b_bytes, bar, keep);
            }
        };
        auto advance = [&](Source& o) {
            o.a += kTma ? 2048 : kABytes;
            o.b += kTma ? 2048u : b_bytes;
            o.ax += 128;
            o.ar += (kTma ? 2048 : kABytes) / kMapRow;
            o.br += static_cast<int>((kTma ? 2048u : b_bytes) / kMapRow);
        };
        // A packed weight does not depend on the kernel before: the weight half of the first stages is requested ahead of the
        // wait, the token half behind it. The raw operator's weight may be that kernel's output, and what it wrote is only
        // sure to be visible behind the wait, also where it let this one in at its end. Device us in a CUDA graph, asked for
        // ahead of the wait / behind it: quant + gemm 4096x12288 128 tokens 14.6 / 14.0, 4096x4096 1 token 8.87 / 8.67;
        // gemm behind gemm 4864x7168 1 token 8.2 / 8.3, 32 tokens 8.0 / 7.8, 1920x11264 1 token 7.5 / 8.1.
        int pre = 0;
        if (!kTma) {
            Walker wa(p, kPair);
            Segment sa;
            uint32_t dst = ring, bar = bar_full;
            while (pre < stages && wa.next(p, sa)) {
                Source o = source(sa);
                for (int kb = sa.k0; kb < sa.k1 && pre < stages; ++kb, ++pre) {
                    if (lead) load_a(o, dst, bar);
                    __syncwarp();
                    advance(o);
                    dst += stage_bytes;
                    bar += 8;
                }
            }
        }
        pdl_wait_prior();
        Walker wk(p, kPair);
        Segment sg;
        int i = 0;
        uint32_t s = 0, phase = 1, dst = ring;        // phase the empty barrier must have completed
        while (!wf.failed && wk.next(p, sg)) {
            Source o = source(sg);
            for (int kb = sg.k0; kb < sg.k1; ++kb, ++i) {
                if (i >= stages && !wf.wait(bar_empty + 8 * s, phase)) break;
                if (lead) {
                    if (i >= pre) load_a(o, dst, bar_full + 8 * s);
                    load_b(o, dst + kABytes, bar_full + 8 * s);
                }
                __syncwarp();
                advance(o);
                dst += stage_bytes;
                if (++s == static_cast<uint32_t>(stages)) { s = 0; phase ^= 1u; dst = ring; }
            }
        }
        if (kPair) {
            // the last stages are handed back by the issuing CTA: this one stays until it has heard of it
            const int last = min(i, stages);
            if (i < stages) { s = 0; phase = 0; }
            for (int j = 0; j < last; ++j) {
                if (!wf.wait(bar_empty + 8 * s, phase)) break;
                if (++s == static_cast<uint32_t>(stages)) { s = 0; phase ^= 1u; }
            }
        }
        if (wf.failed && rank != 0) {                  // let the copies in flight land before the CTA goes: its own are
            for (int j = 0; j < 1000; ++j) __nanosleep(1000);        // counted by the other's barriers, it has none to ask
        } else if (wf.failed)
            for (int j = max(0, i - stages); j < i; ++j) mbar_wait_bounded(bar_full + 8 * (j % stages), (j / stages) & 1, 100000u);
    } else if (warp == 1) {
        // ---------------- MMA issuer -----------------------------------------------------------
        if (kPair && rank != 0) {                      // the other CTA issues for both
        } else if (nch == 1) {
            issue_all<1, kPair>(p, ring, tmem, bar_full, bar_empty, bar_accfull, bar_accempty, wf);
        } else {
            issue_all<2, kPair>(p, ring, tmem, bar_full, bar_empty, bar_accfull, bar_accempty, wf);
        }
    } else {
        // ---------------- epilogue (warps 2..9) ------------------------------------------------
        pdl_wait_prior();                              // out, partials and tickets may still be in use before it
        const int q = warp & 3, half = (warp - 2) >> 2;
        const int row = q * 32 + lane;
        const int cols_half = (((bn >> 4) + 1) >> 1) << 4;
        const int c_lo = half ? cols_half : 0, groups = (half ? bn - cols_half : cols_half) >> 4;
        const bool overlap = acc_overlap(bn) > 0;
        const uintptr_t out_at = reinterpret_cast<uintptr_t>(p.out) | (kDtype == 2 ? 0 : static_cast<uintptr_t>(p.ldc) * 2);
        Store st;
        st.chunk = smem_raw + (ring + stages * stage_bytes - smem_u32(smem_raw)) + half * kStoreChunk;
        st.half = half;
        st.row = row;
        st.align = (out_at & 15) == 0 ? 16 : (out_at & 3) == 0 ? 4 : 2;
        Walker wk(p, kPair);
        Segment sg;
        // Rolled loops of 16 or 32 columns: a tile's columns leave the tensor memory at the pace of the stores. Unrolled over
        // the tile (all of it in registers first) the code was fetched cold once per launch, and 200 registers a thread
        // left no room for these CTAs beside the quantizer's.
        for (int t = 0; wk.next(p, sg); ++t) {
            const int buf = t & 1;
            const int nt = sg.tile / p.tiles_m, mt = sg.tile - nt * p.tiles_m;
            const int n0 = (kPair ? 2 * nt + rank : nt) * kRows, m0 = mt * bn;
            wf.wait(bar_accfull + 8 * buf, (t >> 1) & 1);   // after a time-out: walk on, the warps meet at barriers below
            tc_fence_after();
            const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16) + buf * acc_stride(bn) + c_lo;
            auto release = [&] {                       // the next tile's MMAs may have what was read
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    const uint32_t bar = bar_accempty + (overlap ? 0 : 8 * buf);
                    if (kPair) mbar_arrive_cluster(cluster_map(bar, 0));
                    else mbar_arrive(bar);
                }
            };
            float v[16];
            if (!kPair && p.split > 1) {
                const int S = p.split, w = p.split_cols, part = static_cast<int>(blockIdx.x) % S;
                cluster_sync_all();                    // every CTA of the cluster is through with its ring
#pragma unroll 1
                for (int g = 0; g < groups; ++g) {
                    tmem_ld16(taddr + 16 * g, v);
                    tmem_ld_wait();
                    const int col = c_lo + 16 * g, owner = col / w;
                    const uint32_t dst = cluster_map(ring + ((part * w + col - owner * w) * kRows + row * 4) * 4, owner);
#pragma unroll
                    for (int j = 0; j < 4; ++j) cluster_st16(dst + j * (kRows * 16), v + 4 * j);
                }
                cluster_sync_all();
                const int mine = min(w, bn - part * w);
#pragma unroll 1
                for (int c = 16 * half; c < mine; c += 32) {
                    const float4* src = reinterpret_cast<const float4*>(smem_raw + (ring - smem_u32(smem_raw))) +
                                        (c >> 2) * kRows + row;
#pragma unroll 4
                    for (int r = 0; r < S; ++r) {      // K order
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 x = src[(r * (w >> 2) + j) * kRows];
                            v[4 * j] = r ? v[4 * j] + x.x : x.x;
                            v[4 * j + 1] = r ? v[4 * j + 1] + x.y : x.y;
                            v[4 * j + 2] = r ? v[4 * j + 2] + x.z : x.z;
                            v[4 * j + 3] = r ? v[4 * j + 3] + x.w : x.w;
                        }
                    }
                    store_cols<kDtype, kNMajor, 16>(p, st, n0, m0 + part * w + c, v);
                }
                continue;
            }
            if (kPair || sg.k1 - sg.k0 == p.kblocks) {
                // Whole tile, 32 columns at a time, from the end that the other accumulator overlaps. A half is through with
                // the overlap after `free_at` columns (none: its last tile is drained, this one's need not be); without
                // overlap the accumulator is handed back when all of it has been read.
                const int free_at = !overlap ? 16 * groups : half == buf ? 0 : acc_overlap(bn);
                if (free_at == 0) release();
                int done = 0;
#pragma unroll 1
                while (done < 16 * groups) {
                    const int n = min(32, 16 * groups - done), at = overlap && buf == 0 ? 16 * groups - done - n : done;
                    float u[32];
                    tmem_ld16(taddr + at, u);
                    if (n == 32) tmem_ld16(taddr + at + 16, u + 16);
                    tmem_ld_wait();
                    if (done < free_at && done + n >= free_at) release();
                    done += n;
                    if (kPair && n0 >= p.N) continue;
                    if (n == 32) store_cols<kDtype, kNMajor, 32>(p, st, n0, m0 + c_lo + at, u);
                    else store_cols<kDtype, kNMajor, 16>(p, st, n0, m0 + c_lo + at, u);
                }
                continue;
            }
            // stream-K: leave the partial sums, the last CTA of the tile to arrive adds all of them
            const int base = (sg.tile - p.sk_base) * p.kblocks;
            const int first = sk_owner(p, base), last = sk_owner(p, base + p.kblocks - 1);
            auto slot = [&](int c) {                   // CTA c's partial tile: its first or its last segment
                return reinterpret_cast<float4*>(p.partials) +
                       ((2 * static_cast<int64_t>(c) + (sk_start(p, c) >= base ? 0 : 1)) * bn + c_lo) / 4 * kRows + row;
            };
            float4* own = slot(blockIdx.x);
#pragma unroll 1
            for (int g = 0; g < groups; ++g) {
                tmem_ld16(taddr + 16 * g, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    __stcg(own + (4 * g + j) * kRows, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
            }
            release();
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
#pragma unroll 1
                for (int g = 0; g < groups; ++g) {
#pragma unroll 2
                    for (int c = first; c <= last; ++c) {                // K order, this CTA's own among them
                        const float4* src = slot(c) + 4 * g * kRows;
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float4 x = __ldcg(src + j * kRows);
                            v[4 * j] = c != first ? v[4 * j] + x.x : x.x;
                            v[4 * j + 1] = c != first ? v[4 * j + 1] + x.y : x.y;
                            v[4 * j + 2] = c != first ? v[4 * j + 2] + x.z : x.z;
                            v[4 * j + 3] = c != first ? v[4 * j + 3] + x.w : x.w;
                        }
                    }
                    store_cols<kDtype, kNMajor, 16>(p, st, n0, m0 + c_lo + 16 * g, v);
                }
            }
            named_barrier(1, kEpiWarps * 32);          // s_last is written again for the next shared tile
        }
    }
    // the epilogue's two cluster barriers: all warps of all CTAs take part
    if (!kPair && p.split > 1 && warp < 2) {
        cluster_sync_all();
        cluster_sync_all();
    }

    if (wf.failed && lane == 0) report_timeout(&g_large_status, 6);
    tc_fence_before();
    __syncthreads();
    if (kPair) cluster_sync_all();                     // neither leaves while the other may still reach into it
    if (warp == 1) {
        tc_fence_after();
        if (kPair) tmem_dealloc_pair(tmem, kTmemColsL);
        else tmem_dealloc(tmem, kTmemColsL);
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

// Contiguous memory of that many rows of kMapRow bytes, box of whole rows, no swizzle. (Promoted to 256 bytes in L2 the loads cost
// 24576x4096 with 512 tokens 27.4 us, 27.2 so.)
bool row_map(const void* p, int64_t rows, int box_rows, CUtensorMap* out) {
    EncodeFn fn = encode_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {kMapRow / 8, static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {kMapRow};
    const cuuint32_t box[2] = {kMapRow / 8, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, const_cast<void*>(p), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct LargePlan {
    int bn, nch, tiles_m, tiles, kblocks, stages, grid;
    int dp_rounds, sk_base, sk_ctas, split, split_cols;
    bool pair;
    size_t smem, token_bytes, ticket_bytes, partial_bytes;
};

int g_large_bn = 0, g_large_sk = -1, g_large_min_m = 0;

size_t stage_bytes_of(int bn, bool pair = false) { return kABytes + bn * (pair ? 64 : 128) + (bn + 127) / 128 * 2048; }
int ring_stages(int bn, bool pair = false) {
    const int n = static_cast<int>((kSmemBudget - 1024 - kStoreBytes) / stage_bytes_of(bn, pair));
    return n > kMaxStagesL ? kMaxStagesL : n;
}

// Clusters of S one-per-SM CTAs that run at once: an SM of a GPC that is left over takes none (148 SMs: 74 pairs, 33 fours).
int cluster_capacity(int S, int G) {
    static std::atomic<int> known[64][kMaxSplit + 1] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return G / S;
    int n = known[dev][S].load(std::memory_order_relaxed);
    if (n == 0) {
        const auto kern = gemm_large_kernel<false, 0, false, false>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(G / S * S));
        cfg.blockDim = dim3(kThreadsL);
        cfg.dynamicSmemBytes = kSmemBudget;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(S);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBudget) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = G / S;
        }
        known[dev][S].store(n, std::memory_order_relaxed);
    }
    return n;
}

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
        const double floor_ns = static_cast<double>(N) * K * 9 / 16 / kHbmRate, store = kStorePerToken * bn;
        const auto stage_ns = [&](int64_t ctas) {
            const double issue = kStageBase + kStagePerToken * bn + (nch - 1) * kStageChunk;
            return std::max(issue, static_cast<double>(stage_bytes_of(bn)) * std::min<int64_t>(ctas, G) / kL2Rate);
        };
        const double stage = stage_ns(tiles), wait = acc_overlap(bn) > 0 ? kStoreWait : 0.0;
        const int full = static_cast<int>(tiles / G);
        auto consider = [&](int dp, int ctas, int split, double t, bool pair = false) {
            t = std::max(t, floor_ns + store);
            if (t >= best) return;
            best = t;
            found = true;
            plan->bn = bn; plan->nch = nch; plan->tiles_m = tiles_m; plan->tiles = static_cast<int>(tiles);
            plan->kblocks = kblocks; plan->dp_rounds = dp; plan->sk_ctas = ctas;
            plan->pair = pair;
            plan->split = split; plan->split_cols = (bn / 16 + split - 1) / split * 16;
        };
        if (g_large_sk < 0 || g_large_sk == kPairTuning) {
            const int64_t pairs = static_cast<int64_t>(tiles_m) * ((tiles_n + 1) / 2);
            const int at_once = cluster_capacity(2, G), rounds = static_cast<int>((pairs + at_once - 1) / at_once);
            const double bytes = static_cast<double>(stage_bytes_of(bn, true)) * 2 * std::min<int64_t>(pairs, at_once);
            const double block = std::max(kStageBase + kStagePerToken * bn + (nch - 1) * kStageChunk, bytes / kL2Rate);
            consider(rounds, 0, 1, rounds * std::max(kblocks * block, kStoreWarm * bn) + (rounds - 1) * wait + store + kPairFix, true);
        }
        if (g_large_sk <= 0 || (g_large_sk > 1 && g_large_sk <= kMaxSplit && kblocks < g_large_sk)) {
            const int rounds = static_cast<int>((tiles + G - 1) / G);
            consider(rounds, 0, 1, rounds * std::max(kblocks * stage, kStoreWarm * bn) + (rounds - 1) * wait + store);
        }
        for (int S = 2; S <= kMaxSplit && g_large_sk != 0 && g_large_sk != 1; ++S) {
            if (kblocks < S || (g_large_sk > 1 && S != g_large_sk)) continue;
            const int w = (bn / 16 + S - 1) / S * 16, at_once = cluster_capacity(S, G);
            if (static_cast<size_t>(S) * w * kRows * 4 > static_cast<size_t>(ring_stages(bn)) * stage_bytes_of(bn)) continue;
            const int rounds = static_cast<int>((tiles + at_once - 1) / at_once);
            consider(0, 0, S, rounds * ((kblocks + S - 1) / S * stage_ns(tiles * S) + kSplitBase +
                                        bn * (kSplitPerToken + S * kSplitPerPartToken)) + (rounds - 1) * kSecondWave);
        }
        if (g_large_sk == 0 || g_large_sk > 1) continue;
        for (int dp = full; dp >= 0 && dp >= full - 1; --dp) {
            const int64_t rest = tiles - static_cast<int64_t>(dp) * G;
            if (rest <= 0) continue;
            for (int parts = 2; parts <= 9; ++parts) {             // 9: every CTA
                const int64_t want = rest * parts;
                const int ctas = parts == 9 || want > G ? G : static_cast<int>(want);
                if (rest * kblocks < ctas) continue;
                const double share = static_cast<double>(rest) / ctas;                // tiles per CTA
                const double gather = static_cast<double>(ctas) / rest + 1.0;         // parts of a shared tile, about
                consider(dp, ctas, 1, dp * (kblocks * stage + wait) + (share * kblocks + 1.0) * stage_ns(ctas) + store + kFixBase +
                                          gather * kFixPerPart * ((bn + 31) / 32));
                if (ctas == G) break;
            }
        }
    }
    if (!found) return false;
    plan->stages = ring_stages(plan->bn, plan->pair);
    plan->smem = plan->stages * stage_bytes_of(plan->bn, plan->pair) + kStoreBytes + 1024;
    if (plan->pair) {
        plan->tiles = plan->tiles_m * ((tiles_n + 1) / 2);
        plan->grid = 2 * std::min(plan->tiles, cluster_capacity(2, G));
    } else plan->grid = plan->split > 1 ? plan->tiles * plan->split
                 : plan->dp_rounds > 0 && plan->tiles >= G ? G : (plan->dp_rounds > 0 ? plan->tiles : plan->sk_ctas);
    plan->sk_base = plan->sk_ctas > 0 ? plan->dp_rounds * G : plan->tiles;
    plan->token_bytes = (static_cast<size_t>(plan->tiles_m) * kblocks * (plan->bn * 128 + plan->nch * 2048) + 255) / 256 * 256;
    plan->ticket_bytes = plan->sk_ctas ? (static_cast<size_t>(plan->tiles - plan->sk_base) * 4 + 255) / 256 * 256 : 0;
    plan->partial_bytes = static_cast<size_t>(2) * plan->sk_ctas * plan->bn * kRows * 4;
    return true;
}

// A call asks three times (scratch size, its check, launch) and plans once: 0.3 us each. The device is part of the key: two with
// as many SMs need not place as many clusters.
bool plan_large(int M, int N, int K, bool row_major, LargePlan* plan) {
    struct Last { int M, N, K, dev, bn, sk; bool row_major, found; LargePlan plan; };
    static thread_local Last last = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    if (last.M != M || last.N != N || last.K != K || last.dev != dev || last.bn != g_large_bn || last.sk != g_large_sk ||
        last.row_major != row_major) {
        last = Last{M, N, K, dev, g_large_bn, g_large_sk, row_major, false, {}};
        last.found = make_large_plan(M, N, K, row_major, device_sm_count(), &last.plan);
    }
    *plan = last.plan;
    return last.found;
}

constexpr int kInstances = 18;

// p: PairParams where the plan is for pairs.
cudaError_t launch_with_pdl(int form, const LargePlan& plan, const LargeParams* p, cudaStream_t stream) {
    // packed operands, then row-major ones with M-major and with N-major output; bf16, fp16, fp32; by one CTA, by a pair
#define NVFP4R_KERN(...) reinterpret_cast<const void*>(&gemm_large_kernel<__VA_ARGS__>)
#define NVFP4R_FORMS(PAIR)                                                                                                     \
    NVFP4R_KERN(false, 0, false, PAIR), NVFP4R_KERN(false, 1, false, PAIR), NVFP4R_KERN(false, 2, false, PAIR),                 \
    NVFP4R_KERN(true, 0, false, PAIR), NVFP4R_KERN(true, 1, false, PAIR), NVFP4R_KERN(true, 2, false, PAIR),                    \
    NVFP4R_KERN(true, 0, true, PAIR), NVFP4R_KERN(true, 1, true, PAIR), NVFP4R_KERN(true, 2, true, PAIR)
    static const void* const table[kInstances] = {NVFP4R_FORMS(false), NVFP4R_FORMS(true)};
#undef NVFP4R_KERN
#undef NVFP4R_FORMS
    const int instance = form + (plan.pair ? kInstances / 2 : 0);
    const void* kern = table[instance];
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
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (plan.split > 1 || plan.pair) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = static_cast<unsigned>(plan.pair ? 2 : plan.split);
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (gemv_tuning().use_pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = static_cast<unsigned>(n);
    void* args[1] = {const_cast<LargeParams*>(p)};
    return cudaLaunchKernelExC(&cfg, kern, args);
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
    p->split = plan.split; p->split_cols = plan.split_cols;
    p->dp_rounds = plan.dp_rounds; p->sk_base = plan.sk_base; p->sk_ctas = plan.sk_ctas;
    if (plan.sk_ctas > 0) {
        const int total = (plan.tiles - plan.sk_base) * plan.kblocks;
        p->sk_q = total / plan.sk_ctas;
        p->sk_r = total % plan.sk_ctas;
    }
    p->alpha = alpha;
}

}  // namespace

// Tokens from which the packed linear takes it, where the caller can give it scratch: the device's side of the
// choice. Up to 16 tokens the decode kernel makes one pass over the weight as well and needs no second launch; its
// CTAs each quantize the tokens of their K part, which grows with the tokens, while this path pays a few us for
// partial sums where the weight has few row tiles and long rows. Measured in CUDA graphs, us, decode kernel / this one:
//   N >= 6 K       34816x5120: 13 tokens 23.1 / 19.4, 16 tokens 25.7 / 19.3; 12288x2048: 13 tokens 8.2 / 5.9;
//                  but (N >= 16 K) 24576x1024: 13 tokens 6.2 / 6.9, 17 tokens 8.2 / 6.9
//   N >= 1.5 K     12288x4096: 17 tokens 15.6 / 9.4; 10240x5120: 17 tokens 16.3 / 9.7; 6144x4096: 17 tokens 10.3 / 7.4
//   N >= K         4096x4096: 25 tokens 10.2 / 7.0, 32 tokens 11.6 / 7.1
//   below          4096x12288: 17 tokens 12.2 / 10.3, 24 tokens 13.5 / 10.3, 32 tokens 16.2 / 10.3; 1280x5120: 32 tokens 9.9 / 6.9
// The last two lines were drawn before clusters shared a tile (4096x12288, 24 tokens, 15.7 here) and are kept with the answers
// of the query: this kernel gains on its own side of them.
int large_min_m(int N, int K) {
    const int64_t n = N, k = K;
    return n >= 6 * k && n < 16 * k ? 13 : 2 * n >= 3 * k ? 17 : n >= k ? 25 : 33;
}

// What the entry point takes.
bool large_accepts(int M, int N, int K) {
    return N > 0 && K > 0 && N % kRows == 0 && K % 128 == 0 && M >= (g_large_min_m ? g_large_min_m : large_min_m(N, K));
}

bool large_pays(int M, int N, int K) {
    if (!large_accepts(M, N, K)) return false;
    if (g_large_min_m) return true;
    const int G = device_sm_count(), tiles = N / kRows, kblocks = (K + kBK - 1) / kBK;
    // A narrow weight with rows of 31 or 32 K blocks: the longest that ran as whole tiles here before clusters shared
    // them (0.48 us a block), while two launches of the decode kernel give each CTA one block and one token to add up. 33 / 48 / 64
    // tokens then: 640x8192 13.0 / 14.0 / 14.3, here 15.5 / 15.7 / 15.9; 1280x8192 14.3 / 15.5 / 18.6, here 16.0 / 15.9 / 16.2.
    // With clusters 640x8192 takes 7.7 / 7.7 / 8.0 here, 1280x8192 8.2 / 8.2 / 8.1 (and beside the line 1024x7680 33 tokens
    // 14.8 there, 7.8 here, 1792x8320 17.2 and 8.3): the line stays where callers of the query found it.
    if (M <= 64 && kblocks > 30 && kblocks <= 32 && tiles <= (M <= 48 ? 16 : 8)) return false;
    // Up to 16 tokens both kernels are bound by the weight, and here 1 to 1.5 tiles per SM cost two rounds. The line was
    // drawn when a K block took 0.48 us here (24576x4096, 16 tokens 17.4 / 18.5; 20480x2048 9.8 / 10.8; but 24064x2304, where
    // the decode kernel splits K, now 14.8 / 9.9) and is kept with the answers of the query; at 0.24 us a block this kernel
    // gains on its own side of it: 24576x4096, 16 tokens 17.8 / 14.0, 13 tokens 16.2 / 14.0; 24576x2048 10.3 / 9.5; 20480x2048 9.6 / 9.2.
    if (M <= 16 && tiles > G && 2 * tiles < 3 * G) return packed_time_us(M, N, K) > 3.9 + 0.96 * kblocks;
    return true;
}

size_t large_scratch_bytes(int M, int N, int K) {
    LargePlan plan;
    if (!large_accepts(M, N, K) || !plan_large(M, N, K, false, &plan)) return 0;
    return plan.token_bytes + plan.ticket_bytes + plan.partial_bytes;
}

// The host's side: a second launch and the scratch bring a call to 9.4 us or more even where the device needs 5, while
// a call of the decode kernel ends at 6.5. So up to 32 tokens (one launch of it) that kernel keeps what it does in
// less than 11 us (the estimate is good to 4 %); up to 16 tokens, where the device times lie close together, in less
// than 12. Measured, us a call: 8192x2048 20 tokens 11.3 / 9.6, 6144x4096 11.1 / 9.6; 12288x2048 24 tokens 10.4 / 9.5,
// 20 tokens 9.5 / 10.1; 24576x2048 16 tokens 9.9 / 10.6.
constexpr double kLargeCallUs = 11.0, kLargeCallUsFew = 12.0;

int large_route(int M, int N, int K) {
    if (!large_pays(M, N, K)) return NVFP4R_ROUTE_PACKED;
    return g_large_min_m || M > 32 || packed_time_us(M, N, K) >= (M <= 16 ? kLargeCallUsFew : kLargeCallUs) ? NVFP4R_ROUTE_SCRATCH : NVFP4R_ROUTE_SCRATCH_CAPTURED;
}

cudaError_t launch_linear_large(const PackedLinearArgs& g, void* scratch, cudaStream_t stream) {
    LargePlan plan;
    if (!plan_large(g.M, g.N, g.K, false, &plan)) return cudaErrorInvalidConfiguration;
    uint8_t* tokens = static_cast<uint8_t*>(scratch);
    PairParams p = {};
    fill_common(plan, &p, g.out, g.M, g.N, g.K, g.alpha, false);
    p.w = static_cast<const uint8_t*>(g.packed);
    p.x = tokens;
    p.tickets = reinterpret_cast<unsigned*>(tokens + plan.token_bytes);
    p.partials = reinterpret_cast<float*>(tokens + plan.token_bytes + plan.ticket_bytes);
    const unsigned pieces = static_cast<unsigned>((g.K / kBlockElems + 255) / 256);
    const auto quant = [&](auto kern, int rows) {
        return launch_small(kern, dim3(static_cast<unsigned>((g.M + rows - 1) / rows), pieces), 256, stream,
                            static_cast<const __nv_bfloat16*>(g.xb), g.xb_stride, g.M, g.K, g.gs, g.rcp_mode == kRcpExact, tokens,
                            plan.bn, plan.nch, plan.kblocks, p.tickets, plan.tiles - plan.sk_base);
    };
    // One row a CTA while the CTAs fit the device at once, four (and a quarter of the CTAs) beyond.
    cudaError_t e = static_cast<int64_t>(g.M) * pieces <= 4 * device_sm_count() ? quant(quant_pack_kernel<1>, 1)
                                                                             : quant(quant_pack_kernel<4>, 4);
    if (e != cudaSuccess) return e;
    if (plan.pair) {                                   // made while the quantizer is on its way
        const int64_t blocks = static_cast<int64_t>(plan.tiles_m) * plan.kblocks, rows = blocks * (plan.bn * 128 + plan.nch * 2048) / kMapRow;
        if (!row_map(g.packed, static_cast<int64_t>(g.N / kRows) * plan.kblocks * (kABytes / kMapRow), kABytes / kMapRow, &p.map_w) ||
            !row_map(tokens, rows, plan.bn * 64 / kMapRow, &p.map_x) || !row_map(tokens, rows, plan.nch * 2048 / kMapRow, &p.map_xsf))
            return cudaErrorInvalidValue;
    }
    return launch_with_pdl(g.out_dtype, plan, &p, stream);
}

// The raw operator on row-major operands, any number of tokens. The decode-sized kernel keeps the tokens of a K part in
// shared memory and asks for the weight in one 16 KB tensor-map request a stage from a single lane; fp16 N-major output,
// device us, that kernel / this one: 4864x7168 1 token 21.1 / 8.3, 32 tokens 47.4 / 7.8; 4096x4096 1 token 13.7 / 6.8;
// 640x1024 1 token 6.1 / 4.4; 1920x11264 1 token 10.6 / 8.1. With fp32 output it stays up to 32 tokens: there
// nvfp4r_linear_tc, which quantizes the tokens itself, is bound to give the same bits.
// *taken stays false (nothing launched) where the workspace does not hold what this path needs or a tensor map cannot be
// made: the caller's other kernel runs.
cudaError_t launch_gemm_large(const TcLinearArgs& g, cudaStream_t stream, bool* taken) {
    *taken = false;
    LargePlan plan;
    if (g.xb != nullptr || g.M < g_large_min_m || (g.M <= 32 && (tc_tuned() || g.out_dtype == NVFP4R_F32))) return cudaSuccess;
    if (!plan_large(g.M, g.N, g.K, true, &plan)) return cudaSuccess;
    PairParams p = {};
    fill_common(plan, &p, g.out, g.M, g.N, g.K, g.alpha, g.c_n_major);
    if (!code_map(g.w, g.N, g.K, kRows, &p.map_w) || !code_map(g.a_codes, g.M, g.K, plan.pair ? plan.bn / 2 : plan.bn, &p.map_x)) return cudaSuccess;
    if (plan.pair && (!row_map(g.wsf_swizzled, static_cast<int64_t>(g.N / kRows) * p.k64 / 2, 2, &p.map_wsf) ||
                      !row_map(g.a_sf_swizzled, static_cast<int64_t>((g.M + 127) / 128) * p.k64 / 2, 2, &p.map_xsf)))
        return cudaSuccess;
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
    e = launch_with_pdl((g.c_n_major ? 6 : 3) + g.out_dtype, plan, &p, stream);
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
