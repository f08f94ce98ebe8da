// round_div.cuh -- clamp(rint(v / scale)) without a division per element, bit for bit the division's result.
//
// With ri = RN(1 / scale), v ri and RN(v / scale) are both within 1.5 * 2^-23 |v / scale| of each other, so they round to the
// same integer unless v ri lies that close to a half-integer; only then (and for NaN) is the division carried
// out.  Quotients that matter are at most 64 (4 bits) or 256 (8 bits) in magnitude, which makes the distance 2^-16 or
// 2^-14; anything larger is clamped alike on both ways.
// The rounding itself is the addition of 1.5 * 2^23 (FRND and F2I run at a quarter of the rate of an add), in one FMA with the
// product; its low mantissa bits then are the integer.  How far v ri is from it, another FMA, is 1/2 at most, and only the
// largest of a thread's distances is compared: six instructions an element, where a rounded product, clamped, rounded and
// compared on its own took ten.
#pragma once

#include "common.cuh"

namespace luxcuda {

constexpr float ROUND_MAGIC = 12582912.0f;                 // 1.5 * 2^23
constexpr uint32_t ROUND_MAGIC_BITS = 0x4b400000u;

// Whether RN(1 / scale) is accurate: neither it nor the scale is denormal, infinite or NaN.
__device__ __forceinline__ bool round_div_ok(float scale) { return scale >= 0x1p-126f && scale <= 0x1p126f; }

// t[i] = ROUND_MAGIC_BITS + clamp(rint(v[i] / scale), lo, hi) + off, with |lo|, |hi|, |off| <= 128;
// a NaN quotient counts as 0 and a saturating one as the clamp.
template <int BITS, int N>
__device__ __forceinline__ void round_div(const float (&v)[N], float scale, float ri, bool ok, int lo, int hi, int off, uint32_t (&t)[N]) {
    constexpr float NEAR = BITS == 4 ? 0x1p-16f : 0x1p-14f;
    const float add = ROUND_MAGIC + (float)off, flo = add + (float)lo, fhi = add + (float)hi;
    float worst = 0.0f;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const float y = __fmaf_rn(v[i], ri, add);
        const float d = __fmaf_rn(v[i], ri, -__fsub_rn(y, add));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(worst) : "f"(fabsf(d)));
        t[i] = __float_as_uint(fminf(fmaxf(y, flo), fhi));
    }
    const bool clear = ok && worst <= 0.5f - NEAR;            // false for NaN
    if (!clear) {
#pragma unroll
        for (int i = 0; i < N; i++)
            t[i] = ROUND_MAGIC_BITS + (uint32_t)(min(max(__float2int_rz(rintf(__fdiv_rn(v[i], scale))), lo), hi) + off);
    }
}

// Eight values of four bits (0..15 each), the first in the lowest bits; four of eight bits.
__device__ __forceinline__ uint32_t round_div_pack4(const uint32_t (&t)[8]) {
    uint32_t word = t[7];
#pragma unroll
    for (int i = 6; i >= 0; i--) word = word * 16u + t[i];     // sum of (magic + value) 16^i
    return word - ROUND_MAGIC_BITS * 0x11111111u;
}
__device__ __forceinline__ uint32_t round_div_pack8(uint32_t t0, uint32_t t1, uint32_t t2, uint32_t t3) {
    return __byte_perm(__byte_perm(t0, t1, 0x0040), __byte_perm(t2, t3, 0x0040), 0x5410);
}

}  // namespace luxcuda
