// Quantisation of 256-element groups on one warp, shared by the pack kernels and the decode dot kernel: a lane holds 8
// consecutive elements. The fast path covers groups with |x * 10^dp| < 2^23 throughout, the 64-bit path everything else.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.cuh"
#include "quant_bytes.cuh"

namespace bsi {
namespace {

typedef unsigned long long u64;

template <typename T>
__device__ __forceinline__ float to_float(T v) { return static_cast<float>(v); }
template <>
__device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ long long round_half_away(double x) {
    if (x >= 0.0) return static_cast<long long>(floor(x + 0.5));
    return -static_cast<long long>(floor(-x + 0.5));
}

__device__ __forceinline__ u64 uabs(long long v) { return static_cast<u64>(v >= 0 ? v : -v); }

// half_away(double(f) * 10^dp) in integer arithmetic, bit for bit the value the float64 expression
// gives. With f = m * 2^e (m < 2^24) and mult = 10^dp < 2^27 the product m * mult has at most 51
// bits, so the float64 multiply is exact, and so is the + 0.5 before the floor wherever it can change
// the result; half-away rounding of the exact value is (|P| + 2^(s-1)) >> s. NaN gives 0 and
// magnitudes of 2^63 or more saturate, which is what the float64 -> int64 conversion does.
// mult == 0 selects the float64 path (decimal_places outside [0, 8]).
__device__ __forceinline__ long long decimal_round(float f, double dec_scale, uint32_t mult) {
    if (mult == 0u) return round_half_away(static_cast<double>(f) * dec_scale);
    const uint32_t bits = __float_as_uint(f);
    const uint32_t exp = (bits >> 23) & 0xffu;
    uint32_t man = bits & 0x7fffffu;
    const bool neg = (bits >> 31) != 0u;
    u64 mag;
    if (exp == 255u) {
        mag = man ? 0ull : 0x7fffffffffffffffull;
    } else {
        int e;
        if (exp == 0u) {
            e = -149;
        } else {
            man |= 0x800000u;
            e = static_cast<int>(exp) - 150;
        }
        const u64 P = static_cast<u64>(man) * static_cast<u64>(mult);
        if (e >= 0) {
            mag = (e >= 63 || (P >> (63 - e)) != 0ull) ? (P ? 0x7fffffffffffffffull : 0ull) : (P << e);
        } else {
            const int sh = -e;
            mag = sh >= 53 ? 0ull : ((P + (1ull << (sh - 1))) >> sh);
        }
    }
    return neg ? -static_cast<long long>(mag) : static_cast<long long>(mag);
}

__device__ __forceinline__ u64 warp_max_u64(u64 v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const u64 o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o > v ? o : v;
    }
    return v;
}

__device__ __forceinline__ int shift_for(u64 max_abs, int bits) {
    const int width = max_abs ? (64 - __clzll(static_cast<long long>(max_abs))) : 0;
    int shift = width - (bits - 1);
    shift = shift < 0 ? 0 : shift;
    return shift > 62 ? 62 : shift;
}

// Loads the 8 elements [col, col+8) of a row as float; elements at or beyond D read as 0.
template <typename T>
__device__ __forceinline__ void load8(const T* row, int64_t col, int64_t D, bool vec_ok,
                                      float (&f)[8]) {
    if (vec_ok && col + 8 <= D) {
        if constexpr (sizeof(T) == 2) {
            const uint4 raw = *reinterpret_cast<const uint4*>(row + col);
            const T* h = reinterpret_cast<const T*>(&raw);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = to_float(h[e]);
        } else {
            const float4 a = *reinterpret_cast<const float4*>(row + col);
            const float4 b = *(reinterpret_cast<const float4*>(row + col) + 1);
            f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
            f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = (col + e < D) ? to_float(row[col + e]) : 0.0f;
    }
}

// Quantises the lane's 8 integers with `shift` and clamps: one byte each.
__device__ __forceinline__ u64 quantise8(const long long (&v)[8], int shift, int bits) {
    const long long qmax = (1ll << (bits - 1)) - 1ll;
    const long long qmin = -(1ll << (bits - 1));
    const u64 round_add = shift > 0 ? (1ull << (shift - 1)) : 0ull;
    u64 packed = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const u64 uq = (uabs(v[e]) + round_add) >> shift;
        long long q = v[e] < 0 ? -static_cast<long long>(uq) : static_cast<long long>(uq);
        q = q < qmin ? qmin : q;
        q = q > qmax ? qmax : q;
        packed |= (static_cast<u64>(q) & 0xffull) << (8 * e);
    }
    return packed;
}

// ---- fast path: |x * 10^dp| < 2^23 throughout the group ----------------------------------------------------------
// A lane's 8 elements as loaded: one 16-byte vector for 16-bit types, two for float32. Kept in this form until it is
// quantised, so that loads of later units stay in flight.
template <typename T>
struct RawLane {
    static constexpr int kVecs = sizeof(T) == 2 ? 1 : 2;
    uint4 v[kVecs];
    __device__ __forceinline__ void load(const T* p) {
#pragma unroll
        for (int i = 0; i < kVecs; ++i) v[i] = reinterpret_cast<const uint4*>(p)[i];
    }
    // the first n (at most 8) elements at p one by one, zeros behind them
    __device__ __forceinline__ void load_tail(const T* p, int64_t n) {
        using Bits = typename std::conditional<sizeof(T) == 2, unsigned short, unsigned int>::type;
        const Bits* src = reinterpret_cast<const Bits*>(p);
        Bits b[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) b[e] = e < n ? src[e] : static_cast<Bits>(0);
        if constexpr (sizeof(T) == 2) {
            v[0] = make_uint4(b[0] | (static_cast<uint32_t>(b[1]) << 16), b[2] | (static_cast<uint32_t>(b[3]) << 16),
                              b[4] | (static_cast<uint32_t>(b[5]) << 16), b[6] | (static_cast<uint32_t>(b[7]) << 16));
        } else {
            v[0] = make_uint4(b[0], b[1], b[2], b[3]);
            v[kVecs - 1] = make_uint4(b[4], b[5], b[6], b[7]);
        }
    }
    __device__ __forceinline__ void from_floats(const float (&f)[8]) {   // values of type T held as floats
        if constexpr (sizeof(T) == 2) {
            T h[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) h[e] = static_cast<T>(f[e]);
            v[0] = *reinterpret_cast<const uint4*>(h);
        } else {
            v[0] = make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
            v[kVecs - 1] = make_uint4(__float_as_uint(f[4]), __float_as_uint(f[5]), __float_as_uint(f[6]), __float_as_uint(f[7]));
        }
    }
    // Largest |x| of the lane as a bit pattern of T that orders like the value: NaN and inf above every finite value.
    __device__ __forceinline__ uint32_t abs_max() const {
        if constexpr (sizeof(T) == 2) {
            // in the type's own arithmetic, whose absolute value is an operand modifier; NaN wins and comes out canonical
            using P = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
            const P* p = reinterpret_cast<const P*>(&v[0]);
            const P most = __hmax2_nan(__hmax2_nan(__habs2(p[0]), __habs2(p[1])), __hmax2_nan(__habs2(p[2]), __habs2(p[3])));
            const uint32_t m = *reinterpret_cast<const uint32_t*>(&most);
            return max(m & 0xffffu, m >> 16);
        } else {
            const uint4& a = v[0];
            const uint4& b = v[kVecs - 1];
            return most3(most3(most3(a.x, a.y, a.z), a.w, b.x), most3(b.y, b.z, b.w), 0u);
        }
    }
    // The same of float32 by masks and integer maxima, for the row packer: more instructions, but with maxima of three operands
    // large key sets took longer there (16384 x 4096 keys 86.8 -> 88.0 us, 8192 x 8192 87.0 -> 88.1, most others equal), while
    // the chunk packer gains by those (4096 x 16384 queries 74.8 -> 73.0 us).
    __device__ __forceinline__ uint32_t abs_max_masked() const {
        static_assert(sizeof(T) == 4, "two vectors of float32 patterns");
        const uint4& a = v[0];
        const uint4& b = v[kVecs - 1];
        return max(max(max(a.x & 0x7fffffffu, a.y & 0x7fffffffu), max(a.z & 0x7fffffffu, a.w & 0x7fffffffu)),
                   max(max(b.x & 0x7fffffffu, b.y & 0x7fffffffu), max(b.z & 0x7fffffffu, b.w & 0x7fffffffu)));
    }
    // The pattern abs_max() returns as a float.
    static __device__ __forceinline__ float abs_value(uint32_t bits) {
        if constexpr (std::is_same<T, float>::value) return __uint_as_float(bits);
        else if constexpr (std::is_same<T, __half>::value) return __half2float(__ushort_as_half(static_cast<unsigned short>(bits)));
        else return __uint_as_float(bits << 16);
    }
    // The 8 values quantised with the group's shift, one byte each.
    // kClamp = false where the group needs none (needs_clamp).
    template <bool kClamp = true>
    __device__ __forceinline__ u64 quantise(float mult, int shift, int bits) const {
        float inv, c;
        fast_round_consts(shift, inv, c);
        if constexpr (sizeof(T) == 2) {
            uint32_t w[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t p = h == 0 ? v[0].x : v[0].z, q = h == 0 ? v[0].y : v[0].w;
                w[h] = mask_clamp4<kClamp>(mag(p, 0, mult, inv, c), mag(p, 1, mult, inv, c), mag(q, 0, mult, inv, c),
                                   mag(q, 1, mult, inv, c), prmt(p, q, 0xfdb9u), bits);
            }
            return static_cast<u64>(w[0]) | (static_cast<u64>(w[1]) << 32);
        } else {
            uint32_t w[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4& a = v[h == 0 ? 0 : kVecs - 1];
                w[h] = mask_clamp4<kClamp>(fast_magnitude(__uint_as_float(a.x), mult, inv, c), fast_magnitude(__uint_as_float(a.y), mult, inv, c),
                                           fast_magnitude(__uint_as_float(a.z), mult, inv, c), fast_magnitude(__uint_as_float(a.w), mult, inv, c),
                                           prmt(prmt(a.x, a.y, 0x00fbu), prmt(a.z, a.w, 0x00fbu), 0x5410u), bits);
            }
            return static_cast<u64>(w[0]) | (static_cast<u64>(w[1]) << 32);
        }
    }
private:
    // the largest magnitude of three float32 patterns, NaN above all
    static __device__ __forceinline__ uint32_t most3(uint32_t a, uint32_t b, uint32_t c) {
        float d;
        asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(__uint_as_float(a)), "f"(__uint_as_float(b)), "f"(__uint_as_float(c)));
        return __float_as_uint(d);
    }
    static __device__ __forceinline__ uint32_t mag(uint32_t pair, int half, float mult, float inv, float c) {
        if constexpr (std::is_same<T, __half>::value) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&pair));
            return fast_magnitude(half == 0 ? f.x : f.y, mult, inv, c);
        } else {
            return fast_magnitude(__uint_as_float(half == 0 ? pair << 16 : pair & 0xffff0000u), mult, inv, c);
        }
    }
};

// The shift of a group whose largest |x| is amax; -1: NaN, inf or |x * 10^dp| >= 2^23 somewhere, the group needs the
// generic path.
__device__ __forceinline__ int fast_group_shift(float amax, float mult, int bits) {
    return amax * mult < 8388608.0f ? fast_shift(amax, mult, bits) : -1;
}

// One chunk per warp: false when it needs the generic path. Same integers as that path, far fewer instructions.
template <typename T>
__device__ __forceinline__ bool fast_quantise(const RawLane<T>& r, float mult, int bits, int& shift, u64& packed) {
    const float amax = RawLane<T>::abs_value(__reduce_max_sync(0xffffffffu, r.abs_max()));
    shift = fast_group_shift(amax, mult, bits);
    if (shift < 0) return false;
    // one group in a hundred or so has a value at the clamp: the others skip its steps
    if (needs_clamp(amax, mult, shift, bits)) packed = r.template quantise<true>(mult, shift, bits);
    else packed = r.template quantise<false>(mult, shift, bits);
    return true;
}

// Generic quantiser of one chunk without the stores (the multi-destination kernel's fallback).
template <typename T>
__device__ __noinline__ void generic_quantise(uint4 v0, uint4 v1, double dec_scale, uint32_t dec_mult, int bits, int* shift_out,
                                              u64* packed_out) {
    const uint4 raw[2] = {v0, v1};
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = to_float(reinterpret_cast<const T*>(raw)[e]);
    long long v[8];
    u64 mx = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        v[e] = decimal_round(f[e], dec_scale, dec_mult);
        const u64 a = uabs(v[e]);
        mx = a > mx ? a : mx;
    }
    mx = warp_max_u64(mx);
    const int shift = shift_for(mx, bits);
    *shift_out = shift;
    *packed_out = quantise8(v, shift, bits);
}

}  // namespace
}  // namespace bsi
