// NVFP4 W4A4 GEMV for 2 to 8 tokens: CUDA-core decoding, tensor-core sums (mma.sync m16n8k16, f16 operands,
// f32 accumulators).
//
// An e2m1 code times its e4m3 block scale has at most 6 significant bits between 2^-10 and 2688, so it is
// EXACT in f16, for the weight and for the token alike. The scaled values are the MMA's operands and nothing is
// left to do per block: one MMA replaces 16 x 16 x 8 multiply-adds, and the cost per weight byte (one
// conversion and one f16 multiply per two codes) does not depend on the number of tokens.
//
// tcgen05 is no alternative for this entry: its scale operand wants the 128x4-tiled scale layout, the raw
// operator's scales are row-major and belong to the caller, and 128-row tiles leave most SMs without work.
//
// Decomposition. A CTA takes tiles of 16 weight rows, blockIdx.x, + gridDim.x, ...; its warps split K into
// contiguous ranges of 128-element chunks. The order of K inside an MMA is free as long as both operands use
// the same one, so lane 4 g + t loads 16 bytes (32 elements, two blocks) of row g and of row g + 8 straight
// into registers, which feed 8 MMAs; kStages chunks are in flight per warp, across tiles. The tokens are decoded (and, for
// bf16 tokens, quantized) once per CTA into shared memory, 16 bytes per lane and two MMAs without bank conflicts. The
// warps' sums of a tile meet in shared memory and are added in warp order: results are bit-identical run to run.
//
// Bound: with one CTA of 16 warps per SM (24576x8192, 8 tokens) instruction issue: 61 % of the slots, conversion and f16
// pipes first, waits for loads 0.7 of 6.5 stall cycles an instruction; 24576x4096 runs at 3.7 TB/s. With two CTAs of 8
// warps (7168x5120, 2 tokens) waits for loads come first, 2.3 of 7.9, at 44 % of the slots, and the tile count:
// 448 tiles on 296 CTAs leave half of them one tile, the others two. On small weights the launch and the token
// prologue. Measured against the ring kernel (gemv.cu) and, for K % 256 != 0, the
// plain-load fallback, fp16 out, weights cold in L2, us, before -> after:
//   7168x5120     2 tokens 10.8 -> 8.2    4 tokens 15.4 -> 8.8    8 tokens 24.7 -> 10.0
//   640x1024      2 tokens 2.26 -> 1.67                           8 tokens 4.3 -> 1.8
//   24576x4096    2 tokens 23.6 -> 15.3                           8 tokens 60.2 -> 16.8
//   25600x12288   2 tokens 66.8 -> 47.5   4 tokens 95.9 -> 46.2   8 tokens 169 -> 67.2
//   4100x2080     2 tokens 7.1 -> 3.1                             8 tokens 20.8 -> 4.0
// fp32 rel-L2 error against 64 bits, before -> after: 1000x12288 8 tokens 5.2e-8 -> 3.1e-8, 2048x8192 3 tokens
// 4.8e-8 -> 3.3e-8 (with one chain of 8 MMAs per chunk and an fp32 sum over the warps 7.9e-8 and 6.1e-8).
#include "kernels.h"
#include "quant_core.cuh"

namespace nvfp4r {
namespace {

constexpr int kRowsTile = 16;
constexpr int kStages = 4;
constexpr int kChunkElems = 128;
constexpr int kTokens = 8;

struct MmaParams {
    GemvArgs a;
    int units;       // K / 32
    int chunks;      // ceil(K / 128)
    int tiles;       // ceil(N / 16)
};

// 16 codes (8 bytes) and their scale byte pair half -> 8 exact f16x2
__device__ __forceinline__ void decode_scaled(uint32_t lo, uint32_t hi, __half2 scale, uint32_t h[8]) {
    e2m1x8_to_f16x8(lo, h);
    e2m1x8_to_f16x8(hi, h + 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = as_u32(__hmul2(as_half2(h[i]), scale));
}

__device__ __forceinline__ void mma_f16(float c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void store_out(void* out, int dtype, int64_t idx, float v) {
    if (dtype == 0)      static_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
    else if (dtype == 1) static_cast<__half*>(out)[idx] = __float2half_rn(v);
    else                 static_cast<float*>(out)[idx] = v;
}

struct Chunk {
    uint4 c[2];        // codes of rows g and g + 8
    uint32_t s[2];     // their two block scales
};

template <int kW>      // warps: 8 (two CTAs per SM) or 16 (one)
__global__ void __launch_bounds__(kW * 32, 16 / kW)
gemv_mma_kernel(const __grid_constant__ MmaParams p) {
    extern __shared__ __align__(16) uint4 s_x[];               // [chunk][piece 0..3][token][unit 0..3]
    __shared__ float s_part[2][kW][kTokens][kRowsTile];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int M = p.a.M, N = p.a.N;

    // this warp's chunks; a warp without any walks one empty chunk per tile, so that all meet at the barriers
    const int c0 = warp * p.chunks / kW, c1 = (warp + 1) * p.chunks / kW;
    const int per_tile = max(c1 - c0, 1);
    const int my_tiles = (p.tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
    const int total = my_tiles * per_tile;

    int l_tile = blockIdx.x, l_c = 0;                          // next chunk to request
    auto load = [&](Chunk& st) {
        const int u = (c0 + l_c) * 4 + t;
        const bool live = c0 + l_c < c1 && u < p.units;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            st.c[r] = make_uint4(0u, 0u, 0u, 0u);
            st.s[r] = 0u;
            if (live) {
                const int64_t row = min(l_tile * kRowsTile + g + 8 * r, N - 1);        // rows past the end are not stored
                st.c[r] = ldg_stream_16(p.a.w + row * p.a.w_stride_n + u * 16);
                // plain load: the four lanes' 8 bytes are a quarter of a sector whose rest the warp's next chunks take
                st.s[r] = __ldg(reinterpret_cast<const unsigned short*>(p.a.wsf + row * p.a.wsf_stride_n + u * 2));
            }
        }
        if (++l_c == per_tile) { l_c = 0; l_tile += gridDim.x; }
    };

    // Weights do not depend on the preceding kernel.
    Chunk st[kStages];
#pragma unroll
    for (int s = 0; s < kStages; ++s)
        if (s < total) load(st[s]);
    const float gs = p.a.xb != nullptr ? __ldg(p.a.gs) : 1.0f;
    pdl_launch_dependents();
    pdl_wait_prior();

    // Tokens: unit u of token m -> four pieces of 16 bytes; units past K are zero.
    {
        const bool exact = p.a.rcp_mode == kRcpExact;
        const QuantScales q = exact ? make_quant_scales<kRcpExact>(gs) : make_quant_scales<kRcpApprox>(gs);
        const int padded = p.chunks * 4;
        for (int i = tid; i < M * padded; i += kW * 32) {
            const int m = i / padded, u = i - m * padded;
            uint4 codes = make_uint4(0u, 0u, 0u, 0u);
            uint32_t sf = 0u;
            if (u < p.units) {
                if (p.a.xb != nullptr) {
                    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.a.xb) +
                                                                      m * p.a.xb_stride + u * 32);
                    uint32_t lo[2], hi[2];
                    sf = quantize_block16_rt(__ldg(src), __ldg(src + 1), q, exact, lo);
                    sf |= quantize_block16_rt(__ldg(src + 2), __ldg(src + 3), q, exact, hi) << 8;
                    codes = make_uint4(lo[0], lo[1], hi[0], hi[1]);
                } else {
                    codes = ldg_keep_16(p.a.x + m * p.a.x_stride + u * 16);
                    sf = __ldg(reinterpret_cast<const unsigned short*>(p.a.xsf + m * p.a.xsf_stride + u * 2));
                }
            }
            const __half2 sc = as_half2(e4m3x2_to_f16x2(sf));
            uint32_t h[16];
            decode_scaled(codes.x, codes.y, __low2half2(sc), h);
            decode_scaled(codes.z, codes.w, __high2half2(sc), h + 8);
            uint4* dst = s_x + (static_cast<size_t>(u >> 2) * 4 * M + m) * 4 + (u & 3);
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[j * 4 * M] = make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]);
        }
    }
    __syncthreads();

    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int tile = blockIdx.x, c = 0, buf = 0;
    auto consume = [&](const Chunk& k) {
        uint32_t h[2][16];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const __half2 sc = as_half2(e4m3x2_to_f16x2(k.s[r]));
            decode_scaled(k.c[r].x, k.c[r].y, __low2half2(sc), h[r]);
            decode_scaled(k.c[r].z, k.c[r].w, __high2half2(sc), h[r] + 8);
        }
        // (an empty chunk multiplies zeros by the last chunk's tokens)
        // A chunk's MMAs run in four chains of two (shorter dependences, and sums of four are added in fp32 proper:
        // the tensor core's own accumulation truncates).
        float d[4][4] = {};
        const uint4* xp = s_x + (static_cast<size_t>(min(c0 + c, p.chunks - 1)) * 4 * M + g) * 4 + t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 x = g < M ? xp[j * 4 * M] : make_uint4(0u, 0u, 0u, 0u);
            mma_f16(d[j], h[0][4 * j], h[1][4 * j], h[0][4 * j + 1], h[1][4 * j + 1], x.x, x.y);
            mma_f16(d[j], h[0][4 * j + 2], h[1][4 * j + 2], h[0][4 * j + 3], h[1][4 * j + 3], x.z, x.w);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] += (d[0][j] + d[1][j]) + (d[2][j] + d[3][j]);
    };
    for (int it = 0; it < total; it += kStages) {
#pragma unroll
        for (int s = 0; s < kStages; ++s) {
            if (it + s < total) {
                consume(st[s]);
                if (it + s + kStages < total) load(st[s]);
                if (++c == per_tile) {
                    // every warp comes here once per tile; two buffers, so one barrier per tile is enough
                    float (*part)[kTokens][kRowsTile] = s_part[buf];
                    part[warp][2 * t][g] = acc[0];
                    part[warp][2 * t + 1][g] = acc[1];
                    part[warp][2 * t][g + 8] = acc[2];
                    part[warp][2 * t + 1][g + 8] = acc[3];
                    __syncthreads();
                    const int m = tid / kRowsTile, r = tid % kRowsTile, row = tile * kRowsTile + r;
                    if (m < M && row < N) {
                        double sum[2] = {0.0, 0.0};             // fixed order
#pragma unroll
                        for (int w = 0; w < kW; w += 2) {
                            sum[0] += part[w][m][r];
                            sum[1] += part[w + 1][m][r];
                        }
                        store_out(p.a.out, p.a.out_dtype, m * p.a.out_stride + row,
                                  static_cast<float>(sum[0] + sum[1]) * p.a.alpha);
                    }
                    acc[0] = acc[1] = acc[2] = acc[3] = 0.0f;
                    c = 0;
                    tile += gridDim.x;
                    buf ^= 1;
                }
            }
        }
    }
}

constexpr size_t kSmemPerSm = 227 * 1024;
// Two CTAs per SM up to this much shared memory: the loads in flight live in what is left of the 256 KB for
// L1. A single CTA asks for more than half of what an SM can give, or the driver would carve out room for two.
constexpr size_t kTwoCtaSmem = 168 * 1024, kOneCtaSmem = 100 * 1024;
constexpr size_t x_bytes(int M, int K) { return static_cast<size_t>(M) * ((K + kChunkElems - 1) / kChunkElems) * kChunkElems * 2; }
constexpr size_t part_bytes(int warps) { return static_cast<size_t>(2) * warps * kTokens * kRowsTile * 4; }

}  // namespace

bool gemv_mma_supported(const GemvArgs& a) {
    if (a.M < 2 || a.M > kTokens || a.N < 1 || a.K < 32 || a.K % 32 != 0 || a.K > 65536) return false;
    if (a.pro_kind != 0 || a.push_world > 1) return false;
    if ((reinterpret_cast<uintptr_t>(a.w) & 15) || a.w_stride_n % 16 != 0) return false;
    if ((reinterpret_cast<uintptr_t>(a.wsf) & 1) || a.wsf_stride_n % 2 != 0) return false;
    if (a.xb != nullptr) {
        if ((reinterpret_cast<uintptr_t>(a.xb) & 15) || a.xb_stride % 8 != 0) return false;
    } else {
        if ((reinterpret_cast<uintptr_t>(a.x) & 15) || a.x_stride % 16 != 0) return false;
        if ((reinterpret_cast<uintptr_t>(a.xsf) & 1) || a.xsf_stride % 2 != 0) return false;
    }
    return x_bytes(a.M, a.K) + part_bytes(16) + 1024 <= kSmemPerSm;
}

cudaError_t launch_gemv_mma(const GemvArgs& a, cudaStream_t stream) {
    MmaParams p;
    p.a = a;
    p.units = a.K / 32;
    p.chunks = (a.K + kChunkElems - 1) / kChunkElems;
    p.tiles = (a.N + kRowsTile - 1) / kRowsTile;
    size_t smem = x_bytes(a.M, a.K);
    const bool two = 2 * (smem + part_bytes(8) + 1024) <= kTwoCtaSmem;
    if (!two && smem < kOneCtaSmem) smem = kOneCtaSmem;
    const auto kern = two ? gemv_mma_kernel<8> : gemv_mma_kernel<16>;
    static bool attr_done[2][64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_done[two][dev]) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(kSmemPerSm - 1024 - part_bytes(two ? 8 : 16)));
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_done[two][dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    const int resident = device_sm_count() * (two ? 2 : 1);
    cfg.gridDim = dim3(static_cast<unsigned>(p.tiles < resident ? p.tiles : resident));
    cfg.blockDim = dim3(two ? 256 : 512);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gemv_tuning().use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace nvfp4r
