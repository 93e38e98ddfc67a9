// Stand-alone activation quantizer and block-scale layout conversion kernels.
#include "kernels.h"
#include "quant_core.cuh"

namespace nvfp4r {
namespace {

// One CTA per row and 256 blocks of 16 elements, one thread per block: no division in the index, and the four scales of
// a quad of lanes leave as one word of the swizzled layout. Bound: launch and one trip to memory. It is launched
// programmatically itself, but lets nothing in before it has ended: what it writes may be a weight, which the kernels that
// multiply request before they wait for their predecessor, and launch_dependents makes no store visible. Swizzled scales,
// chained in a CUDA graph, us, one thread per scale with 64-bit divisions and a plain launch -> now: 2x12288 1.64 -> 1.44,
// 128x12288 2.32 -> 1.77, 1000x4096 3.79 -> 2.79.
template <int kMode, bool kSwizzled>
__global__ void __launch_bounds__(256)
quant_kernel(const __nv_bfloat16* __restrict__ x, int64_t x_row_stride, int M, int cols, const float* __restrict__ gs_ptr,
             uint8_t* __restrict__ codes, uint8_t* __restrict__ scales, int cols_out, bool words) {
    pdl_wait_prior();
    const int row = blockIdx.x, col = blockIdx.y * blockDim.x + threadIdx.x;
    if (col >= cols_out) return;
    uint32_t sf = 0;                                   // padding of the swizzled layout
    if (row < M && col < cols) {
        const QuantScales q = make_quant_scales<kMode>(__ldg(gs_ptr));
        const uint4* src = reinterpret_cast<const uint4*>(x + row * x_row_stride + static_cast<int64_t>(col) * kBlockElems);
        const uint4 lo = __ldg(src), hi = __ldg(src + 1);
        uint32_t c[2];
        sf = quantize_block16<kMode>(lo, hi, q, c);
        reinterpret_cast<uint2*>(codes)[static_cast<int64_t>(row) * cols + col] = make_uint2(c[0], c[1]);
    }
    if (kSwizzled && words) {                          // scales 4-byte aligned
        const unsigned quad = 0xFu << (threadIdx.x & 28);                  // cols_out % 4 == 0: its four lanes are here
        sf <<= 8 * (col & 3);
        sf |= __shfl_xor_sync(quad, sf, 1);
        sf |= __shfl_xor_sync(quad, sf, 2);
        if ((col & 3) == 0) *reinterpret_cast<uint32_t*>(scales + swizzled_sf_offset(row, col, cols_out)) = sf;
    } else {
        scales[kSwizzled ? swizzled_sf_offset(row, col, cols_out) : static_cast<int64_t>(row) * cols + col] = static_cast<uint8_t>(sf);
    }
}

template <bool kToFlat>
__global__ void __launch_bounds__(256)
sf_layout_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst,
                 int rows, int cols, int rows_padded, int cols_padded) {
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (kToFlat) {
        if (idx >= static_cast<int64_t>(rows) * cols) return;
        const int r = static_cast<int>(idx / cols), c = static_cast<int>(idx % cols);
        dst[idx] = src[swizzled_sf_offset(r, c, cols_padded)];
    } else {
        if (idx >= static_cast<int64_t>(rows_padded) * cols_padded) return;
        const int r = static_cast<int>(idx / cols_padded), c = static_cast<int>(idx % cols_padded);
        const uint8_t v = (r < rows && c < cols) ? src[static_cast<int64_t>(r) * cols + c] : 0;
        dst[swizzled_sf_offset(r, c, cols_padded)] = v;
    }
}

}  // namespace

cudaError_t launch_quant(const void* x, int64_t x_row_stride, int M, int K, const float* gs,
                         void* codes, void* scales, bool swizzled, int rcp_mode,
                         cudaStream_t stream) {
    const int cols = K / kBlockElems;
    const int rows_out = swizzled ? (M + 127) / 128 * 128 : M;
    const int cols_out = swizzled ? (cols + 3) / 4 * 4 : cols;
    if (rows_out <= 0 || cols_out <= 0) return cudaSuccess;
    const int threads = cols_out < 256 ? (cols_out + 31) / 32 * 32 : 256;
    using Kern = void (*)(const __nv_bfloat16*, int64_t, int, int, const float*, uint8_t*, uint8_t*, int, bool);
    const Kern kern = rcp_mode == kRcpExact ? (swizzled ? quant_kernel<kRcpExact, true> : quant_kernel<kRcpExact, false>)
                                            : (swizzled ? quant_kernel<kRcpApprox, true> : quant_kernel<kRcpApprox, false>);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(rows_out), static_cast<unsigned>((cols_out + threads - 1) / threads));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gemv_tuning().use_pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<const __nv_bfloat16*>(x), x_row_stride, M, cols, gs,
                              static_cast<uint8_t*>(codes), static_cast<uint8_t*>(scales), cols_out,
                              (reinterpret_cast<uintptr_t>(scales) & 3) == 0);
}

cudaError_t launch_sf_layout(const void* src, void* dst, int rows, int K, bool to_flat,
                             cudaStream_t stream) {
    const int cols = K / kBlockElems;
    const int rp = (rows + 127) / 128 * 128, cp = (cols + 3) / 4 * 4;
    const int64_t total = to_flat ? static_cast<int64_t>(rows) * cols : static_cast<int64_t>(rp) * cp;
    const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
    if (to_flat)
        sf_layout_kernel<true><<<blocks, 256, 0, stream>>>(
            static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), rows, cols, rp, cp);
    else
        sf_layout_kernel<false><<<blocks, 256, 0, stream>>>(
            static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), rows, cols, rp, cp);
    return cudaGetLastError();
}

}  // namespace nvfp4r
