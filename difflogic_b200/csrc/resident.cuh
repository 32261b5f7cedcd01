// Rows of one block of samples in shared memory: 4, 8 or 16 bytes.  For the two whole-network kernels.
#pragma once
#include "common.cuh"

namespace dl {

template <int WORDS> struct ResRow;
template <> struct ResRow<1> { using type = uint32_t; };
template <> struct ResRow<2> { using type = uint2; };
template <> struct ResRow<4> { using type = uint4; };

__device__ __forceinline__ uint32_t res_and(uint32_t a, uint32_t b, uint32_t i, uint32_t j) { return (a ^ i) & (b ^ j); }
__device__ __forceinline__ uint2 res_and(const uint2 &a, const uint2 &b, uint32_t i, uint32_t j) {
    return make_uint2(res_and(a.x, b.x, i, j), res_and(a.y, b.y, i, j));
}
__device__ __forceinline__ uint4 res_and(const uint4 &a, const uint4 &b, uint32_t i, uint32_t j) {
    return make_uint4(res_and(a.x, b.x, i, j), res_and(a.y, b.y, i, j), res_and(a.z, b.z, i, j), res_and(a.w, b.w, i, j));
}
__device__ __forceinline__ uint32_t res_xor(uint32_t a, uint32_t b) { return a ^ b; }
__device__ __forceinline__ uint2 res_xor(const uint2 &a, const uint2 &b) { return make_uint2(a.x ^ b.x, a.y ^ b.y); }
__device__ __forceinline__ uint4 res_xor(const uint4 &a, const uint4 &b) { return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w); }
__device__ __forceinline__ void res_fill(uint32_t &v, uint32_t m) { v = m; }
__device__ __forceinline__ void res_fill(uint2 &v, uint32_t m) { v = make_uint2(m, m); }
__device__ __forceinline__ void res_fill(uint4 &v, uint32_t m) { v = make_uint4(m, m, m, m); }
// all ones where bit 15 of w is set
__device__ __forceinline__ uint32_t res_mask15(uint32_t w) {
    uint32_t m;
    asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(m) : "r"(w));
    return m;
}

}  // namespace dl
