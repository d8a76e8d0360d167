// Activations of the mat-vec kernels as exact integers: what mv_id.cu and mv_dense.cu share.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

constexpr int MV_NDIG = 4;
// A value is an integer of magnitude <= 2^30 (the top digit stays within +-64) times its block's scale, 2^29 integers to the
// power of two at or below the largest magnitude.
constexpr int MV_BITS = 29;
// The SUB-wide sums (|sum| <= 2^35) enter an f16 product times 2^-20, in three parts of eleven bits: multiples of 2^5, 2^-6 and
// 2^-17.  With one quantum for all sub-blocks the product with the integer mins or scales is exact, a part at a time.
constexpr int MV_PARTS = 3;
constexpr float MV_SUM_UNSCALE = 0x1p20f;
constexpr float MV_OFFSET = 32.f * MV_SUM_UNSCALE; // Q6_K: what the product of scales and sums stands for, in units of the integers

// One 256-wide block of an activation row, by one warp (eight consecutive values per lane): the integers (or their digits), the block's
// scale, and the SUB-wide sums of the integers as f16 parts, most significant first.
struct MvX {
    float4 a, c;
    __device__ __forceinline__ void load(const float *__restrict__ src, bool want, int lane) { // a row not wanted counts as zero
        a = c = make_float4(0.f, 0.f, 0.f, 0.f);
        if (want) {
            a = __ldg(reinterpret_cast<const float4 *>(src + lane * 8));
            c = __ldg(reinterpret_cast<const float4 *>(src + lane * 8) + 1);
        }
    }
};
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
template <int SUB>
__device__ __forceinline__ void mv_integers(const MvX &in, int (&X)[8], float &sx, __half (&part)[MV_PARTS]) {
    const float v[8] = {in.a.x, in.a.y, in.a.z, in.a.w, in.c.x, in.c.y, in.c.z, in.c.w};
    float amax = 0.f; // NaN if any value is: the block's scale, and with it the result, then is NaN too
#pragma unroll
    for (int j = 0; j < 8; j++) amax = max_nan(amax, fabsf(v[j]));
#pragma unroll
    for (int o = 16; o; o >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    // 2^e <= amax < 2^(e + 1); below 2^-97 the scale stays at the smallest normal number, so that its reciprocal exists
    const int e = max((int)(__float_as_uint(amax) >> 23) - 127, -97);
    const float inv = __int_as_float((127 + MV_BITS - e) << 23);
    sx = e == 128 ? amax : __int_as_float((127 - MV_BITS + e) << 23);
    int sum_h = 0, sum_l = 0; // sums of the upper and the lower 15 bits
#pragma unroll
    for (int j = 0; j < 8; j++) X[j] = __float2int_rn(v[j] * inv);
    if (e == 128) { // an infinite value times an infinite scale; the others count nothing beside it
#pragma unroll
        for (int j = 0; j < 8; j++) X[j] = fabsf(v[j]) == INFINITY ? (v[j] > 0.f ? 1 << MV_BITS : -(1 << MV_BITS)) : 0;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
        sum_h += X[j] >> 15;
        sum_l += X[j] & 0x7fff;
    }
#pragma unroll
    for (int o = 1; o < SUB / 8; o <<= 1) {
        sum_h += __shfl_xor_sync(0xffffffffu, sum_h, o);
        sum_l += __shfl_xor_sync(0xffffffffu, sum_l, o);
    }
    const int q0 = (sum_h + (1 << 9)) >> 10, r0 = (sum_h - (q0 << 10)) * (1 << 15) + sum_l; // |sum_h|, sum_l <= 2^20
    const int q1 = (r0 + (1 << 13)) >> 14, r1 = r0 - (q1 << 14);
    part[0] = __float2half_rn((float)q0 * 0x1p5f);
    part[1] = __float2half_rn((float)q1 * 0x1p-6f);
    part[2] = __float2half_rn((float)((r1 + 4) >> 3) * 0x1p-17f);
}
// Base-256 digits of the integers, most significant first, each digit's eight bytes side by side.
__device__ __forceinline__ void mv_bytes(const int (&X)[8], uint2 (&dig)[MV_NDIG]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t y[4];
#pragma unroll
        for (int j = 0; j < 4; j++) y[j] = (uint32_t)(X[4 * h + j] + 0x808080); // the three low digits become plain bytes plus 128
        // byte d of the four values side by side; the 128 comes off again with the sign bit
        const uint32_t d3 = __byte_perm(__byte_perm(y[0], y[1], 0x40), __byte_perm(y[2], y[3], 0x40), 0x5410) ^ 0x80808080u;
        const uint32_t d2 = __byte_perm(__byte_perm(y[0], y[1], 0x51), __byte_perm(y[2], y[3], 0x51), 0x5410) ^ 0x80808080u;
        const uint32_t d1 = __byte_perm(__byte_perm(y[0], y[1], 0x62), __byte_perm(y[2], y[3], 0x62), 0x5410) ^ 0x80808080u;
        const uint32_t d0 = __byte_perm(__byte_perm(y[0], y[1], 0x73), __byte_perm(y[2], y[3], 0x73), 0x5410);
        if (h == 0) { dig[0].x = d0; dig[1].x = d1; dig[2].x = d2; dig[3].x = d3; }
        else { dig[0].y = d0; dig[1].y = d1; dig[2].y = d2; dig[3].y = d3; }
    }
}
template <int SUB>
__device__ __forceinline__ void mv_digits(const MvX &in, uint2 (&dig)[MV_NDIG], float &sx, __half (&part)[MV_PARTS]) {
    int X[8];
    mv_integers<SUB>(in, X, sx, part);
    mv_bytes(X, dig);
}
// weight of digit d (most significant first)
__device__ __forceinline__ float mv_digit_weight(int d) { return d == 0 ? 16777216.f : (d == 1 ? 65536.f : (d == 2 ? 256.f : 1.f)); }

} // namespace
