// Counter-based Gumbel noise and the float order of the samplers (decode_ops.cu, sample_truncated.cu).
#pragma once
#include <cstdint>

namespace nvfp4r {

// Standard Gumbel noise -log(-log(u)) for element i of a row, from a counter-based generator:
// the 64-bit finalizer of splitmix64 over (key + i * odd constant), top 23 bits -> u in (0, 1).
// `key` already mixes the seed, the row and the row's draw counter, so every draw of every row
// uses its own stream and a replayed CUDA graph keeps drawing fresh numbers.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ float gumbel_uniform(unsigned long long key, int i) {
    const unsigned long long r = mix64(key + static_cast<unsigned long long>(i) * 0x9E3779B97F4A7C15ull);
    // 23 bits: (x + 0.5) / 2^23 is exact in fp32 and stays strictly inside (0, 1)
    return (static_cast<float>(static_cast<unsigned>(r >> 41)) + 0.5f) * (1.0f / 8388608.0f);
}
__device__ __forceinline__ float gumbel_of(float u) { return -logf(-logf(u)); }
__device__ __forceinline__ float gumbel_noise(unsigned long long key, int i) { return gumbel_of(gumbel_uniform(key, i)); }
// Key of one draw: mixes the seed, the row and the row's draw counter.
__device__ __forceinline__ unsigned long long gumbel_key(unsigned long long seed, int row, unsigned long long draw) {
    return mix64(seed ^ mix64((static_cast<unsigned long long>(row) << 40) + draw));
}

// Order-preserving map of a float onto an unsigned key (larger value, larger key): the top-k /
// top-p truncation selects on these keys with a radix descent.
__device__ __forceinline__ uint32_t sortable_key(float x) {
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t key) {
    return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

}  // namespace nvfp4r
