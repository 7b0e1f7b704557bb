// fp32 values as pairs of f16 (see umma_pack.cu): device helpers for the kernels that write them.
#pragma once

#include "umma_gemm.h"

namespace rmlk {

constexpr float SPLIT_LO = 2048.f;  // the low part is stored 2^11 times its size

__device__ __forceinline__ uint32_t finite_abs_bits(float x) {
    const uint32_t b = __float_as_uint(x) & 0x7fffffffu;
    return b < 0x7f800000u ? b : 0u;  // infinities and NaNs stay what they are in the high part and do not set the scale
}
// 2^e with max * 2^e in [2^14, 2^15), from the bits of the largest magnitude; e in [-113, 126]
__device__ __forceinline__ int scale_exponent(uint32_t max_bits) {
    if (max_bits == 0) return 0;
    const int e = 14 - (static_cast<int>(max_bits >> 23) - 127);
    return e > 126 ? 126 : e;
}
__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((e + 127) << 23); }

// Low end of a group's range: the smallest of `nonzero_low` over its values is the bits of the smallest magnitude that is not zero, less one.
__device__ __forceinline__ uint32_t nonzero_low(float x) { return (__float_as_uint(x) & 0x7fffffffu) - 1u; }
// Do pairs under one scale hold every value of the group?  Down to 2^-28 of the largest they keep at least 22 bits; below, a value is off by up to
// 2^-50 of the largest.  Where not, the scale that is stored is negative, the number of such values is stored as well, and sums that they could
// show in are formed again from the fp32 operands (umma_gemm_kernel.cuh, repair).
__device__ __forceinline__ bool pairs_hold(uint32_t max_bits, uint32_t low) {
    return low == 0xffffffffu || __uint_as_float(low + 1u) * 268435456.f >= __uint_as_float(max_bits);
}

// a scaled value that pairs do not hold to 22 bits
__device__ __forceinline__ int is_lossy(float scaled) { return scaled != 0.f && fabsf(scaled) < 6.103515625e-5f ? 1 : 0; }  // 2^-14
__device__ __forceinline__ int lossy4(float4 v, float scale) {
    return is_lossy(v.x * scale) + is_lossy(v.y * scale) + is_lossy(v.z * scale) + is_lossy(v.w * scale);
}

// two scaled values -> their high and low parts
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((a - f.x) * SPLIT_LO, (b - f.y) * SPLIT_LO);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void split8(const float (&x)[8], float scale, uint4& hi, uint4& lo) {
    split2(x[0] * scale, x[1] * scale, hi.x, lo.x);
    split2(x[2] * scale, x[3] * scale, hi.y, lo.y);
    split2(x[4] * scale, x[5] * scale, hi.z, lo.z);
    split2(x[6] * scale, x[7] * scale, hi.w, lo.w);
}
// four values of row m at column k (a multiple of 4)
__device__ __forceinline__ void store_pairs4(const SplitRows& d, int64_t m, int64_t k, float4 v, float scale) {
    uint2 hi, lo;
    split2(v.x * scale, v.y * scale, hi.x, lo.x);
    split2(v.z * scale, v.w * scale, hi.y, lo.y);
    __half* p = static_cast<__half*>(d.data) + m * d.k_pad + k;
    *reinterpret_cast<uint2*>(p) = hi;
    *reinterpret_cast<uint2*>(p + d.m_pad * d.k_pad) = lo;
}
// the same values in fp32, for a row that pairs do not hold
__device__ __forceinline__ void store_full4(const SplitRows& d, int64_t m, int64_t k, float4 v) { *reinterpret_cast<float4*>(d.full + m * d.full_ld + k) = v; }

}  // namespace rmlk
