// Device helpers shared by the pack kernels and the re-quantising linear epilogue: the exact float32 form of the
// reference's two roundings and the byte-wise sign / clamp.
#pragma once

#include <stdint.h>

namespace bsi {

// prmt.b32 with the full 4-bit selectors (values 8..15 replicate the sign bit of the chosen byte over the
// result byte; the __byte_perm intrinsic only honours 3 bits per selector).
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// u0..u3 carry the unsigned quantised magnitudes of four elements in their low bytes (0 .. 2^(bits-1)), m is 0xff in
// the bytes of the negative ones. Clamps positives to 2^(bits-1)-1 (kClamp: some may be beyond), negates the negatives
// and returns the four two's-complement bytes.
template <bool kClamp>
__device__ __forceinline__ uint32_t mask_clamp4(uint32_t u0, uint32_t u1, uint32_t u2, uint32_t u3, uint32_t m, int bits) {
    uint32_t w = __byte_perm(__byte_perm(u0, u1, 0x0040), __byte_perm(u2, u3, 0x0040), 0x5410);   // the low bytes
    if (kClamp) {
        // positive 2^(bits-1) -> 2^(bits-1) - 1 (the byte is exactly `top` there, so the borrow stays inside it)
        const uint32_t over = w & ~m & (0x01010101u << (bits - 1));
        w -= over >> (bits - 1);
    }
    // negate the bytes under m: (~b + 1) per byte, the carry kept inside the byte by adding in 7 bits. Without a
    // magnitude of 128 the top bit of w ^ m is m's.
    const uint32_t t = ((w ^ m) & 0x7f7f7f7fu) + (m & 0x01010101u);
    return kClamp ? t ^ ((w ^ m) & 0x80808080u) : t ^ (m & 0x80808080u);
}

// The reference's two roundings, |v| = floor(|x| * 10^dp + 0.5) and (|v| + [shift > 0] * 2^(shift-1)) >> shift, as two
// FMAs with round toward zero. An FMA rounds the exact product and sum once, so no operand width matters:
//   r1 = fma_rz(|x|, mult, 2^22 + 0.5)   floats in [2^22, 2^23) are the multiples of 1/2 and those in [2^23, 2^24) the
//                                        integers, so the truncation leaves 2^22 + |v| + h/2 with h in {0, 1}
//   u  = fma_rz(r1, 2^-shift, c)         c = 2^23 + [shift > 0] / 2 - 2^(22-shift), exact in float32 for shift <= 23:
//                                        2^23 + the wanted integer (h/2 never reaches the next one), truncated
// Valid while |x| * mult < 2^23; mult = 10^dp is exact in float32 up to 10^10.
__device__ __forceinline__ float fast_round1(float abs_x, float mult) { return __fmaf_rz(abs_x, mult, 4194304.5f); }

// Shift of a group whose largest |x| is amax (amax * mult < 2^23): bits(max|v|) - (b - 1), clamped at 0.
__device__ __forceinline__ int fast_shift(float amax, float mult, int bits) {
    const uint32_t mx = __float2uint_rz(fast_round1(amax, mult) - 4194304.0f);   // the difference is exact
    const int shift = (32 - __clz(static_cast<int>(mx))) - (bits - 1);
    return shift < 0 ? 0 : shift;
}

// Constants of the second rounding for a given shift.
__device__ __forceinline__ void fast_round_consts(int shift, float& inv, float& c) {
    inv = __uint_as_float(static_cast<uint32_t>(127 - shift) << 23);   // 2^-shift
    c = (8388608.0f - 4194304.0f * inv) + (shift > 0 ? 0.5f : 0.0f);   // both steps exact
}

// Whether a group with largest magnitude amax holds values beyond the clamp, i.e. amax itself rounds to 2^(bits-1).
__device__ __forceinline__ bool needs_clamp(float amax, float mult, int shift, int bits) {
    float inv, c;
    fast_round_consts(shift, inv, c);
    return (__float_as_uint(__fmaf_rz(fast_round1(amax, mult), inv, c)) & 0xffu) >> (bits - 1) != 0u;
}

// Quantised magnitude of x in the low mantissa byte of the result.
__device__ __forceinline__ uint32_t fast_magnitude(float x, float mult, float inv, float c) {
    return __float_as_uint(__fmaf_rz(fast_round1(fabsf(x), mult), inv, c));
}

}  // namespace bsi
