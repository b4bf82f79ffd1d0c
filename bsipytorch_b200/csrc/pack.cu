// Fused quantise + bit-slice pack kernels (queries: per-256-element chunk scale; keys: per-row
// scale), the slice -> int8 recombination, and the cast+bias layer epilogue.
//
// One warp owns one 256-element chunk of one row: lane L holds elements 8L..8L+7, read with one
// 16-byte (f16/bf16) or two 16-byte (f32) loads, so a warp reads 512 B / 1 KiB contiguously.
// The largest |v| of the chunk is reduced with shuffles, the 8 clamped values of a lane are
// bit-transposed in registers (8x8), and byte s of the result is the lane's byte of slice s:
// byte (L % 8) of word (L / 8) of the chunk. The int8 image is written 8 bytes per lane.
//
// Arithmetic follows the reference bit for bit (bsi_cuda_kernels_quant.cuh:24-29, 82-108,
// 291-341, 414-488): v = half_away(double(float(x)) * 10^dp); bits = 64 - clz(max|v|);
// shift = clamp(bits - (b-1), 0, 62); q = sign(v) * ((|v| + (shift ? 1 << (shift-1) : 0)) >> shift),
// clamped to [-2^(b-1), 2^(b-1)-1].
#include "quantise.cuh"

namespace bsi {
namespace {

__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Shift selection with outlier clipping (bsi_cuda_kernels_quant.cuh:82-108, BSI_FIXED_CLIP_K > 0): the width comes
// from min(max |v|, clip_k * mean |v|) instead of max |v|, so a few extreme values no longer push the whole group
// to a coarse shift; they saturate at the clamp instead. `sum_abs` is the sum of the group's |v| (integers, so any
// summation order gives the same double below 2^53), `count` its number of elements.
__device__ __forceinline__ int shift_for_clipped(u64 max_abs, double sum_abs, int count, int bits, float clip_k) {
    int width = 0;
    if (count > 0) {
        double effective = static_cast<double>(max_abs);
        const double clip_max = (sum_abs / static_cast<double>(count)) * static_cast<double>(clip_k);
        if (clip_max < effective) effective = clip_max;
        if (effective > 0.0) (void)frexp(effective, &width);
    } else {
        width = max_abs ? (64 - __clzll(static_cast<long long>(max_abs))) : 0;
    }
    int shift = width - (bits - 1);
    shift = shift < 0 ? 0 : shift;
    return shift > 62 ? 62 : shift;
}

// Transposes the 8x8 bit matrix held in x (row e = byte e, LSB first): afterwards bit e of
// byte s is the former bit s of byte e.
__device__ __forceinline__ u64 transpose8x8(u64 x) {
    u64 t;
    t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAull;
    x = x ^ t ^ (t << 7);
    t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCull;
    x = x ^ t ^ (t << 14);
    t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ull;
    x = x ^ t ^ (t << 28);
    return x;
}

// The same transposition on the two 32-bit halves (lo = rows 0..3, hi = rows 4..7): the first two exchange steps
// stay inside a half, the third swaps the high nibbles of lo with the low nibbles of hi.
__device__ __forceinline__ void transpose8x8_halves(uint32_t& lo, uint32_t& hi) {
    uint32_t t;
    t = (lo ^ (lo >> 7)) & 0x00AA00AAu;  lo ^= t * 0x81u;       // t ^ (t << 7) on the multiplier: the logic pipe is the
    t = (hi ^ (hi >> 7)) & 0x00AA00AAu;  hi ^= t * 0x81u;       // one these kernels fill
    t = (lo ^ (lo >> 14)) & 0x0000CCCCu; lo ^= t * 0x4001u;
    t = (hi ^ (hi >> 14)) & 0x0000CCCCu; hi ^= t * 0x4001u;
    t = (lo ^ (hi << 4)) & 0xF0F0F0F0u;
    lo ^= t;
    hi ^= t >> 4;
}

// Writes the lane's 8 clamped values (one byte each in `packed`): int8 image and bit slices.
__device__ __forceinline__ void store_packed(u64 packed, int bits, int lane, int64_t chunk, int64_t W,
                                             u64* __restrict__ words_row, int8_t* __restrict__ q8_row) {
    if (q8_row != nullptr) {
        *reinterpret_cast<u64*>(q8_row + chunk * 256 + lane * 8) = packed;
    }
    if (words_row != nullptr) {
        const int64_t word = chunk * 4 + (lane >> 3);
        if (word < W) {
            const u64 t = transpose8x8(packed);
            uint8_t* dst = reinterpret_cast<uint8_t*>(words_row + word) + (lane & 7);
            const uint32_t tl = static_cast<uint32_t>(t), th = static_cast<uint32_t>(t >> 32);
            const size_t step = static_cast<size_t>(W) * 8u;
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                if (s < bits) dst[s * step] = static_cast<uint8_t>((s < 4 ? tl : th) >> (8 * (s & 3)));
            }
        }
    }
}

__device__ __forceinline__ void emit_chunk(const long long (&v)[8], int shift, int bits, int lane,
                                           int64_t chunk, int64_t W, u64* __restrict__ words_row,
                                           int8_t* __restrict__ q8_row) {
    store_packed(quantise8(v, shift, bits), bits, lane, chunk, W, words_row, q8_row);
}

// One (row, chunk) unit on the generic path (any decimal_places, any magnitude, NaN/inf, any layout):
// 64-bit integers and 64-bit offsets throughout.
template <typename T>
__device__ __forceinline__ void generic_unit(const T* x, int64_t unit, int64_t D, int64_t ldx,
                                             double dec_scale, uint32_t dec_mult, int bits, int64_t chunks, int64_t W,
                                             u64* __restrict__ words, float* __restrict__ scales,
                                             int32_t* __restrict__ shifts, int8_t* __restrict__ q8, int64_t ld8,
                                             bool vec, int lane, float clip_k = 0.0f,
                                             float* __restrict__ sq_norms = nullptr) {
    // no sum of squares from this path: infinity makes a dot's exactness test that reads it fail safely
    if (sq_norms != nullptr && lane == 0) sq_norms[unit] = __int_as_float(0x7f800000);
    const int64_t row = unit / chunks;
    const int64_t chunk = unit - row * chunks;
    float f[8];
    load8<T>(x + row * ldx, chunk * 256 + lane * 8, D, vec, f);
    long long v[8];
    u64 mx = 0;
    double sum = 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        v[e] = decimal_round(f[e], dec_scale, dec_mult);
        const u64 a = uabs(v[e]);
        mx = a > mx ? a : mx;
        sum += static_cast<double>(a);     // elements beyond D were loaded as 0
    }
    mx = warp_max_u64(mx);
    int shift;
    if (clip_k > 0.0f) {
        const int64_t left = D - chunk * 256;
        shift = shift_for_clipped(mx, warp_sum_f64(sum), static_cast<int>(left < 256 ? left : 256), bits, clip_k);
    } else {
        shift = shift_for(mx, bits);
    }
    if (lane == 0) {
        if (scales != nullptr) scales[unit] = static_cast<float>(1ull << shift);
        if (shifts != nullptr) shifts[unit] = shift;
    }
    emit_chunk(v, shift, bits, lane, chunk, W, words != nullptr ? words + row * bits * W : nullptr,
               q8 != nullptr ? q8 + row * ld8 : nullptr);
}

// Chunk mode without preconditions: one warp per unit, grid-stride.
template <typename T>
__global__ void __launch_bounds__(256) quantize_pack_chunk_generic_kernel(
    const T* __restrict__ x, int64_t rows, int64_t D, int64_t ldx, double dec_scale, uint32_t dec_mult, int bits,
    int64_t chunks, int64_t W, u64* __restrict__ words, float* __restrict__ scales,
    int32_t* __restrict__ shifts, int8_t* __restrict__ q8, int64_t ld8, int vec_ok, float clip_k,
    float* __restrict__ sq_norms) {
    const int lane = threadIdx.x & 31;
    const int64_t total = rows * chunks;
    for (int64_t unit = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); unit < total;
         unit += static_cast<int64_t>(gridDim.x) * 8)
        generic_unit<T>(x, unit, D, ldx, dec_scale, dec_mult, bits, chunks, W, words, scales, shifts, q8, ld8,
                        vec_ok != 0, lane, clip_k, sq_norms);
}

// After the 8x8 bit transposition a lane holds one byte of each slice. Four neighbouring lanes (half a 64-bit word)
// trade bytes in two shuffle steps so that each ends up with the four bytes of two slices, first_slice(lane) and the
// one after it: two 4-byte stores per lane instead of seven 1-byte stores.
__device__ __forceinline__ int first_slice(int lane) { return ((lane & 2) << 1) + ((lane & 1) << 1); }
__device__ __forceinline__ void slice_pieces(u64 packed, int lane, uint32_t& w0, uint32_t& w1) {
    uint32_t tl = static_cast<uint32_t>(packed), th = static_cast<uint32_t>(packed >> 32);
    transpose8x8_halves(tl, th);
    const bool upper = (lane & 2) != 0;     // lanes 2, 3 of the group collect slices 4..7, lanes 0, 1 slices 0..3
    const bool odd = (lane & 1) != 0;       // odd lanes keep the second slice pair of their group
    const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? tl : th, 2);
    const uint32_t x = upper ? got : tl;    // the slice group's bytes of group lane (lane & 1)
    const uint32_t y = upper ? th : got;    // ... and of group lane (lane & 1) + 2
    const uint32_t keep = __byte_perm(x, y, odd ? 0x7632 : 0x5410);
    const uint32_t other = __shfl_xor_sync(0xffffffffu, __byte_perm(x, y, odd ? 0x5410 : 0x7632), 1);
    w0 = __byte_perm(keep, other, odd ? 0x2604 : 0x6240);   // bytes of group lanes 0, 1, 2, 3
    w1 = __byte_perm(keep, other, odd ? 0x3715 : 0x7351);
}

// +-2^i with the top slice negative (bsi_cuda.cpp:217-236), times the row scale where there is one
__device__ __forceinline__ float slice_weight(int slice, int bits, float scale) {
    const float w = __uint_as_float(static_cast<uint32_t>(127 + slice) << 23) * scale;
    return slice == bits - 1 ? -w : w;
}

// Fast path of one chunk including its stores: true when the chunk was quantised and stored.
template <typename T, bool kWords, bool kQ8>
__device__ __forceinline__ bool fast_chunk(const RawLane<T>& r, uint32_t unit, uint32_t q8_off, uint32_t word_off,
                                           bool word_ok, int lane, float mult, int bits, uint32_t slice_bytes,
                                           u64* __restrict__ words, float* __restrict__ scales,
                                           int32_t* __restrict__ shifts, int8_t* __restrict__ q8,
                                           float* __restrict__ sq_norms) {
    int shift;
    u64 packed;
    if (!fast_quantise<T>(r, mult, bits, shift, packed)) return false;
    if (sq_norms != nullptr) {
        // sum of squares of the chunk's de-shifted integers, (2^shift)^2 * sum a^2: an exact float (the integer
        // sum is at most 256 * 128^2 = 2^22), which a dot's exactness test turns into a Cauchy-Schwarz bound
        int n2 = __dp4a(static_cast<int>(static_cast<uint32_t>(packed)), static_cast<int>(static_cast<uint32_t>(packed)), 0);
        n2 = __dp4a(static_cast<int>(static_cast<uint32_t>(packed >> 32)), static_cast<int>(static_cast<uint32_t>(packed >> 32)), n2);
        n2 = __reduce_add_sync(0xffffffffu, n2);
        if (lane == 0) sq_norms[unit] = static_cast<float>(n2) * __uint_as_float(static_cast<uint32_t>(127 + 2 * shift) << 23);
    }
    if (lane == 0) {
        scales[unit] = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);   // 2^shift
        if (shifts != nullptr) shifts[unit] = shift;
    }
    if constexpr (kQ8) *reinterpret_cast<u64*>(q8 + q8_off) = packed;
    if constexpr (kWords) {
        uint32_t w0, w1;
        slice_pieces(packed, lane, w0, w1);
        if (word_ok) {
            const int s0 = first_slice(lane);
            uint8_t* out = reinterpret_cast<uint8_t*>(words);
            // word_off addresses the lane's own byte (word lane / 8, byte lane % 8); the 4-byte store goes to
            // the start of its half word
            const uint32_t off = word_off - (lane & 3) + static_cast<uint32_t>(s0) * slice_bytes;
            if (s0 < bits) *reinterpret_cast<uint32_t*>(out + off) = w0;
            if (s0 + 1 < bits) *reinterpret_cast<uint32_t*>(out + off + slice_bytes) = w1;
        }
    }
    return true;
}

#ifndef BSI_PACK_MIN_BLOCKS
#define BSI_PACK_MIN_BLOCKS 4
#endif

// Geometry of a fast chunk-mode launch; the host checks that every offset fits 32 bits.
struct FastGeom {
    uint32_t total, chunks, D, ldx, ld8, W;
    uint32_t row_bytes;     // bits * W * 8: bytes of one row's slices
    uint32_t slice_bytes;   // W * 8
};

constexpr int kSlowQueue = 8;   // units per warp that may wait for the generic path

// Persistent fast chunk kernel. The grid is sized to what is resident at once and every warp walks the (row, chunk)
// units with stride gridDim.x * 8, kDepth units' loads in flight: at 32 warps per SM one unit of a 16-bit type is 16 KB
// per SM, and HBM at full rate needs 40 KB and more in flight per SM. Units the fast path cannot take are queued and
// redone on the generic path after the loop, which keeps the 64-bit code out of the loop's register budget; a warp
// whose queue overflows redoes all of its units.
// kDense: x and q8 are contiguous (ldx == ld8 == D), D is a multiple of 256 and x is 16-byte aligned, so
// a unit's element offset is unit * 256 and no lane ever needs the scalar tail loads.
template <typename T, bool kDense, bool kWords, bool kQ8>
__global__ void __launch_bounds__(256, BSI_PACK_MIN_BLOCKS) quantize_pack_chunk_fast_kernel(
    const T* x, FastGeom g, double dec_scale, uint32_t dec_mult, int bits,
    u64* __restrict__ words, float* __restrict__ scales, int32_t* __restrict__ shifts, int8_t* __restrict__ q8,
    int vec_ok, float* __restrict__ sq_norms, float* __restrict__ slice_weights) {
    // Launched as a programmatic dependent, and letting its own dependents go at once: a dot sets up its barriers and
    // tensor memory while this kernel runs, and reads its results behind griddepcontrol.wait.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    x = behind_wait(x);
    __shared__ uint32_t slow_queue[8][kSlowQueue];
    constexpr int kDepth = sizeof(T) == 2 ? 4 : 2;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const uint32_t stride = gridDim.x * 8u;
    const uint32_t first = blockIdx.x * 8u + warp;
    if (kWords && slice_weights != nullptr) {   // in chunk mode a row's slice weights do not depend on its values
        const uint32_t n = (g.total / g.chunks) * static_cast<uint32_t>(bits);
        for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u)
            slice_weights[i] = slice_weight(static_cast<int>(i % static_cast<uint32_t>(bits)), bits, 1.0f);
    }
    if (first >= g.total) return;
    constexpr bool kRows = !kDense || kWords;   // row / chunk are needed, not just the unit number
    const uint32_t stride_rows = kRows ? stride / g.chunks : 0u;
    const uint32_t stride_chunks = kRows ? stride - stride_rows * g.chunks : 0u;
    const float mult = static_cast<float>(dec_mult);
    const bool vec = kDense || vec_ok != 0;
    const uint32_t lane_col = lane * 8u;
    const uint32_t lane_word = (lane >> 3) * 8u + (lane & 7u);   // byte within the chunk's 4 words
    int nslow = 0;

    struct Pos { uint32_t unit, row, chunk; };
    auto advance = [&](Pos& p) {
        p.unit += stride;
        if constexpr (kRows) {
            p.row += stride_rows; p.chunk += stride_chunks;
            if (p.chunk >= g.chunks) { p.chunk -= g.chunks; ++p.row; }
        }
    };
    auto fetch = [&](RawLane<T>& r, const Pos& p) {
        if constexpr (kDense) {
            r.load(x + (p.unit * 256u + lane_col));
        } else {
            const uint32_t col = p.chunk * 256u + lane_col;
            const T* src = x + static_cast<int64_t>(p.row) * g.ldx;
            if (vec && col + 8u <= g.D) r.load(src + col);
            else r.load_tail(src + (col < g.D ? col : 0u), static_cast<int64_t>(g.D) - static_cast<int64_t>(col));
        }
    };

    Pos cur, nxt;
    cur.unit = first;
    cur.row = kRows ? first / g.chunks : 0u;
    cur.chunk = kRows ? first - cur.row * g.chunks : 0u;
    nxt = cur;
    RawLane<T> buf[kDepth];
#pragma unroll
    for (int j = 0; j < kDepth; ++j) {
        if (nxt.unit < g.total) fetch(buf[j], nxt);
        advance(nxt);
    }
    while (cur.unit < g.total) {
#pragma unroll
        for (int j = 0; j < kDepth; ++j) {
            if (cur.unit < g.total) {
                const RawLane<T> r = buf[j];
                if (nxt.unit < g.total) fetch(buf[j], nxt);
                const uint32_t q8_off = kDense ? cur.unit * 256u + lane_col : cur.row * g.ld8 + cur.chunk * 256u + lane_col;
                const uint32_t word_off = kWords ? cur.row * g.row_bytes + cur.chunk * 32u + lane_word : 0u;
                const bool word_ok = kDense || cur.chunk * 4u + (lane >> 3) < g.W;
                if (!fast_chunk<T, kWords, kQ8>(r, cur.unit, q8_off, word_off, word_ok, lane, mult, bits, g.slice_bytes,
                                                words, scales, shifts, q8, sq_norms)) {
                    if (nslow < kSlowQueue && lane == 0) slow_queue[warp][nslow] = cur.unit;
                    ++nslow;
                }
                advance(cur);
                advance(nxt);
            }
        }
    }
    if (nslow == 0) return;
    __syncwarp();
    const int64_t ld8 = kDense ? g.D : g.ld8;
    if (nslow <= kSlowQueue) {
        for (int i = 0; i < nslow; ++i)
            generic_unit<T>(x, slow_queue[warp][i], g.D, g.ldx, dec_scale, dec_mult, bits, g.chunks, g.W, words, scales,
                            shifts, q8, ld8, vec, lane, 0.0f, sq_norms);
    } else {
        for (uint32_t unit = first; unit < g.total; unit += stride)
            generic_unit<T>(x, unit, g.D, g.ldx, dec_scale, dec_mult, bits, g.chunks, g.W, words, scales, shifts, q8,
                            ld8, vec, lane, 0.0f, sq_norms);
    }
}

// Two units per warp at a time, for 16-bit types: a lane holds 16 consecutive elements, lanes 0 to 15 those of one unit, 16 to 31
// those of the next. The kernel above is bound by instruction issue (178 a unit with slices, 117 without), and a third of
// them do not depend on how many elements a lane has: maximum, shift, rounding constants, addresses, the loop. Here they are
// paid once per two units, the int8 image leaves 16 bytes per lane, and two lanes instead of four trade the slices' bytes
// (4096 x 16384 float16: 60.7 -> 52.4 us with slices).
// For more units than warps are resident; below that the kernel above spreads them over twice the warps.
template <typename T, bool kDense, bool kWords, bool kQ8>
__global__ void __launch_bounds__(256, BSI_PACK_MIN_BLOCKS) quantize_pack_chunk_pair_kernel(
    const T* x, FastGeom g, double dec_scale, uint32_t dec_mult, int bits,
    u64* __restrict__ words, float* __restrict__ scales, int32_t* __restrict__ shifts, int8_t* __restrict__ q8,
    int vec_ok, float* __restrict__ sq_norms, float* __restrict__ slice_weights) {
    static_assert(sizeof(T) == 2, "16 elements are two 16-byte vectors");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // as above
    asm volatile("griddepcontrol.wait;" ::: "memory");
    x = behind_wait(x);
    __shared__ uint32_t slow_queue[8][kSlowQueue];
    constexpr int kDepth = 2;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const bool upper = lane >= 16;                    // the second unit's lanes
    const uint32_t l = lane & 15u;
    const uint32_t stride = gridDim.x * 16u;
    const uint32_t first = (blockIdx.x * 8u + warp) * 2u;
    if (kWords && slice_weights != nullptr) {         // in chunk mode a row's slice weights do not depend on its values
        const uint32_t n = (g.total / g.chunks) * static_cast<uint32_t>(bits);
        for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u)
            slice_weights[i] = slice_weight(static_cast<int>(i % static_cast<uint32_t>(bits)), bits, 1.0f);
    }
    if (first >= g.total) return;
    constexpr bool kRows = !kDense || kWords;
    const uint32_t stride_rows = kRows ? stride / g.chunks : 0u;
    const uint32_t stride_chunks = kRows ? stride - stride_rows * g.chunks : 0u;
    const float mult = static_cast<float>(dec_mult);
    const bool vec = kDense || vec_ok != 0;
    const uint32_t lane_col = l * 16u;
    int nslow = 0;

    struct Pos { uint32_t unit, row, chunk; };        // of the lane's unit
    struct Raw { RawLane<T> a, b; };
    auto advance = [&](Pos& p) {
        p.unit += stride;
        if constexpr (kRows) {
            p.row += stride_rows; p.chunk += stride_chunks;
            if (p.chunk >= g.chunks) { p.chunk -= g.chunks; ++p.row; }
        }
    };
    auto fetch = [&](Raw& r, const Pos& p) {
        if (p.unit >= g.total) {                      // the last pair of an odd number of units
            r.a.v[0] = r.b.v[0] = make_uint4(0u, 0u, 0u, 0u);
        } else if constexpr (kDense) {
            const T* src = x + (p.unit * 256u + lane_col);
            r.a.load(src);
            r.b.load(src + 8);
        } else {
            const uint32_t col = p.chunk * 256u + lane_col;
            const T* src = x + static_cast<int64_t>(p.row) * g.ldx;
            const int64_t left = static_cast<int64_t>(g.D) - static_cast<int64_t>(col);
            if (vec && left >= 16) {
                r.a.load(src + col);
                r.b.load(src + col + 8);
            } else {
                r.a.load_tail(src + (left > 0 ? col : 0u), left);
                r.b.load_tail(src + (left > 8 ? col + 8u : 0u), left - 8);
            }
        }
    };
    auto process = [&](const Raw& r, const Pos& p) {
        const uint32_t m = max(r.a.abs_max(), r.b.abs_max());
        const uint32_t m0 = __reduce_max_sync(0xffffffffu, upper ? 0u : m), m1 = __reduce_max_sync(0xffffffffu, upper ? m : 0u);
        const float amax = RawLane<T>::abs_value(upper ? m1 : m0);
        const int shift = fast_group_shift(amax, mult, bits);
        const bool there = p.unit < g.total;
        const uint32_t slow = __ballot_sync(0xffffffffu, there && shift < 0);
        if (slow != 0u) {                             // NaN, infinity, beyond 2^23: either unit may be one
            if (slow & 1u) {
                if (nslow < kSlowQueue && lane == 0) slow_queue[warp][nslow] = p.unit;
                ++nslow;
            }
            if (slow >> 31) {
                if (nslow < kSlowQueue && lane == 31) slow_queue[warp][nslow] = p.unit;
                ++nslow;
            }
        }
        const bool store = there && shift >= 0;
        // one group in a hundred or so has a value at the clamp: the others skip its steps
        u64 pa, pb;
        if (__any_sync(0xffffffffu, store && needs_clamp(amax, mult, shift, bits))) {
            pa = r.a.template quantise<true>(mult, shift, bits);
            pb = r.b.template quantise<true>(mult, shift, bits);
        } else {
            pa = r.a.template quantise<false>(mult, shift, bits);
            pb = r.b.template quantise<false>(mult, shift, bits);
        }
        uint32_t al = static_cast<uint32_t>(pa), ah = static_cast<uint32_t>(pa >> 32), bl = static_cast<uint32_t>(pb), bh = static_cast<uint32_t>(pb >> 32);
        if (sq_norms != nullptr) {                    // see fast_chunk
            int n2 = __dp4a(static_cast<int>(al), static_cast<int>(al), __dp4a(static_cast<int>(ah), static_cast<int>(ah), 0));
            n2 = __dp4a(static_cast<int>(bl), static_cast<int>(bl), __dp4a(static_cast<int>(bh), static_cast<int>(bh), n2));
            const int n0 = __reduce_add_sync(0xffffffffu, upper ? 0 : n2), n1 = __reduce_add_sync(0xffffffffu, upper ? n2 : 0);
            if (store && l == 0) sq_norms[p.unit] = static_cast<float>(upper ? n1 : n0) * __uint_as_float(static_cast<uint32_t>(127 + 2 * shift) << 23);
        }
        if (store && l == 0) {
            scales[p.unit] = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);   // 2^shift
            if (shifts != nullptr) shifts[p.unit] = shift;
        }
        if constexpr (kQ8) {
            const uint32_t q8_off = kDense ? p.unit * 256u + lane_col : p.row * g.ld8 + p.chunk * 256u + lane_col;
            if (store) *reinterpret_cast<uint4*>(q8 + q8_off) = make_uint4(al, ah, bl, bh);
        }
        if constexpr (kWords) {
            transpose8x8_halves(al, ah);              // byte s: the lane's first eight bits of slice s (ah: slices 4 to 7)
            transpose8x8_halves(bl, bh);              // ... and its next eight
            // even lanes collect slices 0 to 3 of both lanes of their pair, odd lanes slices 4 to 7
            const bool odd = (lane & 1) != 0;
            const uint32_t ga = __shfl_xor_sync(0xffffffffu, odd ? al : ah, 1), gb = __shfl_xor_sync(0xffffffffu, odd ? bl : bh, 1);
            const uint32_t ka = odd ? ah : al, kb = odd ? bh : bl;
            const uint32_t a0 = odd ? ga : ka, b0 = odd ? gb : kb, a1 = odd ? ka : ga, b1 = odd ? kb : gb;      // even lane's, odd lane's
            const uint32_t e0 = __byte_perm(a0, b0, 0x5140), e2 = __byte_perm(a0, b0, 0x7362);      // slice s: bytes a, b; then slice s + 1
            const uint32_t o0 = __byte_perm(a1, b1, 0x5140), o2 = __byte_perm(a1, b1, 0x7362);
            if (store && p.chunk * 4u + (l >> 2) < g.W) {
                const int s0 = odd ? 4 : 0;
                uint8_t* out = reinterpret_cast<uint8_t*>(words) +
                               (p.row * g.row_bytes + p.chunk * 32u + (l & 14u) * 2u + static_cast<uint32_t>(s0) * g.slice_bytes);
                if (s0 < bits) *reinterpret_cast<uint32_t*>(out) = __byte_perm(e0, o0, 0x5410);
                if (s0 + 1 < bits) *reinterpret_cast<uint32_t*>(out + g.slice_bytes) = __byte_perm(e0, o0, 0x7632);
                if (s0 + 2 < bits) *reinterpret_cast<uint32_t*>(out + 2u * g.slice_bytes) = __byte_perm(e2, o2, 0x5410);
                if (s0 + 3 < bits) *reinterpret_cast<uint32_t*>(out + 3u * g.slice_bytes) = __byte_perm(e2, o2, 0x7632);
            }
        }
    };

    Pos cur, nxt;
    cur.unit = first + (upper ? 1u : 0u);
    cur.row = kRows ? cur.unit / g.chunks : 0u;
    cur.chunk = kRows ? cur.unit - cur.row * g.chunks : 0u;
    nxt = cur;
    Raw buf[kDepth];
#pragma unroll
    for (int j = 0; j < kDepth; ++j) {
        fetch(buf[j], nxt);
        advance(nxt);
    }
    const uint32_t end = g.total + (upper ? 1u : 0u);       // a warp stays together: its first unit decides
    while (cur.unit < end) {
#pragma unroll
        for (int j = 0; j < kDepth; ++j) {
            if (cur.unit < end) {
                const Raw r = buf[j];
                fetch(buf[j], nxt);
                process(r, cur);
                advance(cur);
                advance(nxt);
            }
        }
    }
    if (nslow == 0) return;
    __syncwarp();
    const int64_t ld8 = kDense ? g.D : g.ld8;
    if (nslow <= kSlowQueue) {
        for (int i = 0; i < nslow; ++i)
            generic_unit<T>(x, slow_queue[warp][i], g.D, g.ldx, dec_scale, dec_mult, bits, g.chunks, g.W, words, scales,
                            shifts, q8, ld8, vec, lane, 0.0f, sq_norms);
    } else {
        for (uint32_t unit = first; unit < g.total; unit += stride)
            for (uint32_t u = unit; u < min(unit + 2u, g.total); ++u)
                generic_unit<T>(x, u, g.D, g.ldx, dec_scale, dec_mult, bits, g.chunks, g.W, words, scales, shifts, q8,
                                ld8, vec, lane, 0.0f, sq_norms);
    }
}

// The same for what a query batch and a layer ask for (int8 image, scales and sums of squares; kWords: slices and their weights)
// of rows of whole chunks on 16-byte vectors. The kernel above is bound by instruction issue (167 a unit, 77 % of the slots), so a
// warp takes G turns of two units each of one row here: all loads go out together, addresses are a base and an immediate, and
// nothing is asked per unit that the launch knows. 4096 x 16384 float16 with slices 51.1 -> 45.9 us (5.7 TB/s, 88 % of the copy rate),
// 512 x 8192 5.5 -> 4.6. (float32, one unit per turn: 65.6 -> 63.6 us with slices, 71 -> 74 without; not built.)
template <typename T, int G, bool kWords>
__global__ void __launch_bounds__(256, 4) quantize_pack_chunk_turns_kernel(
    const T* x, uint32_t rows, uint32_t per_row /* warps */, uint32_t chunks, double dec_scale, uint32_t dec_mult, int bits,
    u64* __restrict__ words, float* __restrict__ scales, int8_t* __restrict__ q8, float* __restrict__ sq_norms,
    float* __restrict__ slice_weights) {
    static_assert(sizeof(T) == 2, "16 elements are two 16-byte vectors");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // as above
    asm volatile("griddepcontrol.wait;" ::: "memory");
    x = behind_wait(x);
    const int lane = threadIdx.x & 31;
    const bool upper = lane >= 16;                        // the second unit's lanes
    const uint32_t l = lane & 15u;
    const uint32_t item = blockIdx.x * 8u + (threadIdx.x >> 5);
    const uint32_t row = item / per_row, c0 = (item - row * per_row) * (2u * G);       // first chunk
    if (kWords) {                                         // in chunk mode a row's slice weights do not depend on its values
        const uint32_t n = rows * static_cast<uint32_t>(bits);
        for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u)
            slice_weights[i] = slice_weight(static_cast<int>(i % static_cast<uint32_t>(bits)), bits, 1.0f);
    }
    if (row >= rows) return;
    const uint32_t D = chunks * 256u, W = chunks * 4u;
    const int turns = static_cast<int>(min((chunks - c0 + 1u) / 2u, static_cast<uint32_t>(G)));
    const uint32_t chunk = c0 + (upper ? 1u : 0u);        // the lane's, in turn 0
    const size_t at = static_cast<size_t>(row) * D + chunk * 256u + l * 16u;
    const float mult = static_cast<float>(dec_mult);
    struct Raw { RawLane<T> a, b; };
    Raw raw[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
        if (i < turns && chunk + 2u * i < chunks) {
            raw[i].a.load(x + at + i * 512);
            raw[i].b.load(x + at + i * 512 + 8);
        } else {
            raw[i].a.v[0] = raw[i].b.v[0] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    int8_t* q8_out = q8 + at;
    float* scale_out = scales + (row * chunks + chunk);
    float* sq_out = sq_norms + (row * chunks + chunk);
    const uint32_t slice_words = 2u * W;                  // 32-bit words per slice
    const bool odd = (lane & 1) != 0;                     // even lanes collect slices 0 to 3 of both lanes of their pair, odd lanes 4 to 7
    const int s0 = odd ? 4 : 0;
    uint32_t* w_out = nullptr;
    if (kWords) w_out = reinterpret_cast<uint32_t*>(words + (static_cast<size_t>(row) * bits + s0) * W) + chunk * 8u + (l >> 1);
    uint32_t slow = 0;                                    // bit i: turn i has a unit of the 64-bit path; bit 16 + i: the lane's is one
#pragma unroll
    for (int i = 0; i < G; ++i) {
        if (i >= turns) break;
        const Raw& r = raw[i];
        const uint32_t m = max(r.a.abs_max(), r.b.abs_max());
        const uint32_t m0 = __reduce_max_sync(0xffffffffu, upper ? 0u : m), m1 = __reduce_max_sync(0xffffffffu, upper ? m : 0u);
        const float amax = RawLane<T>::abs_value(upper ? m1 : m0);
        const int shift = fast_group_shift(amax, mult, bits);
        const bool there = chunk + 2u * i < chunks;
        const bool store = there && shift >= 0;
        if (__any_sync(0xffffffffu, there && shift < 0)) slow |= (1u << i) | (there && shift < 0 ? 0x10000u << i : 0u);
        u64 pa, pb;
        if (__any_sync(0xffffffffu, store && needs_clamp(amax, mult, shift, bits))) {      // one group in a hundred or so
            pa = r.a.template quantise<true>(mult, shift, bits);
            pb = r.b.template quantise<true>(mult, shift, bits);
        } else {
            pa = r.a.template quantise<false>(mult, shift, bits);
            pb = r.b.template quantise<false>(mult, shift, bits);
        }
        uint32_t al = static_cast<uint32_t>(pa), ah = static_cast<uint32_t>(pa >> 32), bl = static_cast<uint32_t>(pb), bh = static_cast<uint32_t>(pb >> 32);
        int n2 = __dp4a(static_cast<int>(al), static_cast<int>(al), __dp4a(static_cast<int>(ah), static_cast<int>(ah), 0));      // see fast_chunk
        n2 = __dp4a(static_cast<int>(bl), static_cast<int>(bl), __dp4a(static_cast<int>(bh), static_cast<int>(bh), n2));
        const int n0 = __reduce_add_sync(0xffffffffu, upper ? 0 : n2), n1 = __reduce_add_sync(0xffffffffu, upper ? n2 : 0);
        if (store && l == 0u) {
            scale_out[i * 2] = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);      // 2^shift
            sq_out[i * 2] = static_cast<float>(upper ? n1 : n0) * __uint_as_float(static_cast<uint32_t>(127 + 2 * shift) << 23);
        }
        if (store) *reinterpret_cast<uint4*>(q8_out + i * 512) = make_uint4(al, ah, bl, bh);
        if constexpr (kWords) {
            transpose8x8_halves(al, ah);                  // as in the kernel above
            transpose8x8_halves(bl, bh);
            const uint32_t ga = __shfl_xor_sync(0xffffffffu, odd ? al : ah, 1), gb = __shfl_xor_sync(0xffffffffu, odd ? bl : bh, 1);
            const uint32_t ka = odd ? ah : al, kb = odd ? bh : bl;
            const uint32_t a0 = odd ? ga : ka, b0 = odd ? gb : kb, a1 = odd ? ka : ga, b1 = odd ? kb : gb;
            const uint32_t e0 = __byte_perm(a0, b0, 0x5140), e2 = __byte_perm(a0, b0, 0x7362);
            const uint32_t o0 = __byte_perm(a1, b1, 0x5140), o2 = __byte_perm(a1, b1, 0x7362);
            if (store) {
                uint32_t* w = w_out + i * 16;
                if (s0 < bits) w[0] = __byte_perm(e0, o0, 0x5410);
                if (s0 + 1 < bits) w[slice_words] = __byte_perm(e0, o0, 0x7632);
                if (s0 + 2 < bits) w[2u * slice_words] = __byte_perm(e2, o2, 0x5410);
                if (s0 + 3 < bits) w[3u * slice_words] = __byte_perm(e2, o2, 0x7632);
            }
        }
    }
    if ((slow & 0xffffu) == 0u) return;
#pragma unroll 1
    for (int u = 0; u < 2 * turns; ++u)
        if (__shfl_sync(0xffffffffu, slow, (u & 1) * 16) & (0x10000u << (u >> 1)))
            generic_unit<T>(x, static_cast<int64_t>(row) * chunks + c0 + u, D, D, dec_scale, dec_mult, bits, chunks, W, kWords ? words : nullptr,
                            scales, nullptr, q8, D, true, lane, 0.0f, sq_norms);
}

// Destinations of the multi-destination pack: the same int8 image / chunk scales go to each of them.
struct MultiDst {
    int n_q8, n_scales;
    int8_t* q8[BSI_B200_MAX_PEERS];
    float* scales[BSI_B200_MAX_PEERS];
};

// Chunk-mode pack whose int8 image and chunk scales are stored to several destinations at once (own
// memory and peer mappings alike): element (row, col) at q8[i] + row * ld8 + col, the scale of
// (row, chunk) at scales[i] + row * scale_ld + chunk. Persistent warps with next-unit prefetch as in
// the fast kernel; D is a multiple of 256 and x is 16-byte aligned, so every lane loads vectors.
template <typename T>
__global__ void __launch_bounds__(256, BSI_PACK_MIN_BLOCKS) quantize_pack_multi_kernel(
    const T* __restrict__ x, uint32_t total, uint32_t chunks, uint32_t ldx, uint32_t ld8, uint32_t scale_ld,
    double dec_scale, uint32_t dec_mult, int bits, const MultiDst dst) {
    const int lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * 8u;
    const uint32_t first = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (first >= total) return;
    const uint32_t stride_rows = stride / chunks;
    const uint32_t stride_chunks = stride - stride_rows * chunks;
    const uint32_t lane_col = lane * 8u;
    const bool try_fast = dec_mult != 0u;

    struct Pos { uint32_t unit, row, chunk; };
    auto advance = [&](Pos p) {
        p.unit += stride; p.row += stride_rows; p.chunk += stride_chunks;
        if (p.chunk >= chunks) { p.chunk -= chunks; ++p.row; }
        return p;
    };
    auto fetch = [&](RawLane<T>& r, const Pos& p) { r.load(x + (p.row * ldx + p.chunk * 256u + lane_col)); };
    auto process = [&](const RawLane<T>& r, const Pos& p) {
        int shift;
        u64 packed;
        if (!(try_fast && fast_quantise<T>(r, static_cast<float>(dec_mult), bits, shift, packed)))
            generic_quantise<T>(r.v[0], r.v[RawLane<T>::kVecs - 1], dec_scale, dec_mult, bits, &shift, &packed);
        const uint32_t q8_off = p.row * ld8 + p.chunk * 256u + lane_col;
        const uint32_t sc_off = p.row * scale_ld + p.chunk;
        const float scale = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);   // 2^shift, shift <= 62
#pragma unroll
        for (int i = 0; i < BSI_B200_MAX_PEERS; ++i) {
            if (i < dst.n_q8) *reinterpret_cast<u64*>(dst.q8[i] + q8_off) = packed;
            if (i < dst.n_scales && lane == 0) dst.scales[i][sc_off] = scale;
        }
    };

    Pos cur;
    cur.unit = first;
    cur.row = first / chunks;
    cur.chunk = first - cur.row * chunks;
    RawLane<T> a, b;
    fetch(a, cur);
    for (;;) {
        Pos nxt = advance(cur);
        bool more = nxt.unit < total;
        if (more) fetch(b, nxt);
        process(a, cur);
        if (!more) break;
        cur = nxt;
        nxt = advance(cur);
        more = nxt.unit < total;
        if (more) fetch(a, nxt);
        process(b, cur);
        if (!more) break;
        cur = nxt;
    }
}

// Residual add + LayerNorm + activation pack of one token row per block, for 16-bit layer types:
//   x_out = T(x + delta)                      (delta may be null: x_out = x)
//   y     = T((x_out - mean) * rstd * gamma + beta), float32 statistics over the row (two passes over registers)
//   y is quantised per 256-element chunk exactly as the chunk-mode packer would quantise it and the int8
//   image / chunk scales go to the destinations (own buffer or peer mappings), as in the multi-destination pack.
// Warp w owns chunks w, w + 8, ...; lane L the 8 consecutive elements 8L..8L+7 of each (the packer's mapping), so the
// row stays in registers between the add, the statistics and the quantisation. CPW = chunks per warp (H <= 2048*CPW).
template <typename T, int CPW>
__global__ void __launch_bounds__(256) add_layernorm_pack_kernel(
    const T* __restrict__ x, const T* __restrict__ delta, const T* __restrict__ gamma, const T* __restrict__ beta,
    float eps, int rows, int H, int chunks, T* __restrict__ x_out, double dec_scale, uint32_t dec_mult,
    int bits, int64_t ld8, int64_t scale_ld, const MultiDst dst) {
    __shared__ float red[2][8];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const bool try_fast = dec_mult != 0u;
    const float inv_h = 1.0f / static_cast<float>(H);
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        const int64_t base = static_cast<int64_t>(row) * H;
        float v[CPW][8];
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            const int c = warp + i * 8;
            if (c < chunks) {
                const int64_t off = base + c * 256 + lane * 8;
                uint4 raw = __ldg(reinterpret_cast<const uint4*>(x + off));
                const T* xv = reinterpret_cast<const T*>(&raw);
                if (delta != nullptr) {
                    const uint4 draw = __ldg(reinterpret_cast<const uint4*>(delta + off));
                    const T* dv = reinterpret_cast<const T*>(&draw);
                    T ov[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        ov[e] = static_cast<T>(to_float(xv[e]) + to_float(dv[e]));
                        v[i][e] = to_float(ov[e]);
                    }
                    *reinterpret_cast<uint4*>(x_out + off) = *reinterpret_cast<const uint4*>(ov);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[i][e] = to_float(xv[e]);
                    if (x_out != x) *reinterpret_cast<uint4*>(x_out + off) = raw;
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) sum += v[i][e];
            }
        }
        // mean
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) red[0][warp] = sum;
        __syncthreads();
        float tot = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) tot += red[0][w];
        const float mean = tot * inv_h;
        // variance around the mean
        float sq = 0.0f;
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            if (warp + i * 8 < chunks) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float d = v[i][e] - mean;
                    sq = fmaf(d, d, sq);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (lane == 0) red[1][warp] = sq;
        __syncthreads();
        float tsq = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) tsq += red[1][w];
        const float rstd = rsqrtf(tsq * inv_h + eps);
        // normalise, round to the layer type, quantise the chunk, store everywhere
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
            const int c = warp + i * 8;
            if (c < chunks) {
                const int col = c * 256 + lane * 8;
                const uint4 graw = __ldg(reinterpret_cast<const uint4*>(gamma + col));
                const uint4 braw = __ldg(reinterpret_cast<const uint4*>(beta + col));
                const T* gv = reinterpret_cast<const T*>(&graw);
                const T* bv = reinterpret_cast<const T*>(&braw);
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    f[e] = to_float(static_cast<T>(fmaf((v[i][e] - mean) * rstd, to_float(gv[e]), to_float(bv[e]))));
                RawLane<T> r;
                r.from_floats(f);
                int shift;
                u64 packed;
                if (!(try_fast && fast_quantise<T>(r, static_cast<float>(dec_mult), bits, shift, packed)))
                    generic_quantise<T>(r.v[0], r.v[RawLane<T>::kVecs - 1], dec_scale, dec_mult, bits, &shift, &packed);
                const int64_t q8_off = static_cast<int64_t>(row) * ld8 + col;
                const int64_t sc_off = static_cast<int64_t>(row) * scale_ld + c;
                const float scale = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);
#pragma unroll
                for (int d = 0; d < BSI_B200_MAX_PEERS; ++d) {
                    if (d < dst.n_q8) *reinterpret_cast<u64*>(dst.q8[d] + q8_off) = packed;
                    if (d < dst.n_scales && lane == 0) dst.scales[d][sc_off] = scale;
                }
            }
        }
        __syncthreads();   // red[] is rewritten by the next row
    }
}

// ---- variable-slice mode (no shift: the decimal integers themselves are sliced) ---------------------------------
// Pass 1: largest |v| and "has a negative" per row, v = half_away(double(float(x)) * 10^dp). The reference takes
// them with torch reductions over the int64 tensor (bsi_vector_cuda.cpp:1089-1099, 1156-1159).
template <typename T>
__global__ void __launch_bounds__(256) decimal_absmax_kernel(const T* __restrict__ x, int64_t rows, int64_t D, int64_t ldx,
                                                             double dec_scale, uint32_t dec_mult, int64_t chunks, int vec_ok,
                                                             u64* __restrict__ row_absmax, int32_t* __restrict__ row_negative) {
    __shared__ u64 wmax[8];
    __shared__ int wneg[8];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int64_t row = blockIdx.x;
    const T* xr = x + row * ldx;
    u64 mx = 0;
    int neg = 0;
    for (int64_t chunk = warp; chunk < chunks; chunk += 8) {
        float f[8];
        load8<T>(xr, chunk * 256 + lane * 8, D, vec_ok != 0, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const long long v = decimal_round(f[e], dec_scale, dec_mult);
            const u64 a = uabs(v);
            mx = a > mx ? a : mx;
            neg |= v < 0 ? 1 : 0;
        }
    }
    mx = warp_max_u64(mx);
    neg = __any_sync(0xffffffffu, neg) ? 1 : 0;
    if (lane == 0) {
        wmax[warp] = mx;
        wneg[warp] = neg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        u64 m = 0;
        int n = 0;
        for (int w = 0; w < 8; ++w) {
            m = wmax[w] > m ? wmax[w] : m;
            n |= wneg[w];
        }
        row_absmax[row] = m;
        row_negative[row] = n;
    }
}

// Pass 2: the low `slices` bits of the two's-complement integers as bit slices (what launch_pack_bits_all_ballot_batch
// writes, bsi_cuda_kernels_pack.cuh:129-174, 204-230), plus, for the tensor-core dot, the integers as two signed
// 8-bit digits: v = 128 * hi + lo with lo in [0, 127] (hi8 may be NULL when every |v| <= 127: lo8 then holds v itself).
// One warp per 256-element chunk, lane = 8 elements, byte (lane % 8) of word (lane / 8) of each slice.
template <typename T>
__global__ void __launch_bounds__(256) pack_plain_kernel(const T* __restrict__ x, int64_t rows, int64_t D, int64_t ldx,
                                                         double dec_scale, uint32_t dec_mult, int slices, int64_t chunks,
                                                         int64_t W, int vec_ok, u64* __restrict__ words,
                                                         int8_t* __restrict__ lo8, int8_t* __restrict__ hi8, int64_t ld8) {
    const int lane = threadIdx.x & 31;
    const int64_t unit = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (unit >= rows * chunks) return;
    const int64_t row = unit / chunks;
    const int64_t chunk = unit - row * chunks;
    float f[8];
    load8<T>(x + row * ldx, chunk * 256 + lane * 8, D, vec_ok != 0, f);
    long long v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = decimal_round(f[e], dec_scale, dec_mult);
    if (lo8 != nullptr) {
        u64 lo = 0, hi = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (hi8 != nullptr) {
                lo |= static_cast<u64>(v[e] & 127) << (8 * e);
                hi |= static_cast<u64>((v[e] >> 7) & 255) << (8 * e);
            } else {
                lo |= static_cast<u64>(v[e] & 255) << (8 * e);
            }
        }
        *reinterpret_cast<u64*>(lo8 + row * ld8 + chunk * 256 + lane * 8) = lo;
        if (hi8 != nullptr) *reinterpret_cast<u64*>(hi8 + row * ld8 + chunk * 256 + lane * 8) = hi;
    }
    if (words != nullptr) {
        const int64_t word = chunk * 4 + (lane >> 3);
        if (word < W) {
            uint8_t* base = reinterpret_cast<uint8_t*>(words + (row * slices) * W + word) + (lane & 7);
            for (int s = 0; s < slices; ++s) {
                uint32_t byte = 0;
#pragma unroll
                for (int e = 0; e < 8; ++e) byte |= static_cast<uint32_t>((v[e] >> s) & 1ll) << e;
                base[static_cast<int64_t>(s) * W * 8] = static_cast<uint8_t>(byte);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) quantize_pack_row_kernel(
    const T* __restrict__ x, int64_t rows, int64_t D, int64_t ldx, double dec_scale, uint32_t dec_mult, int bits,
    int64_t chunks, int64_t W, u64* __restrict__ words, float* __restrict__ scales,
    int32_t* __restrict__ shifts, int8_t* __restrict__ q8, int64_t ld8, int vec_ok, float clip_k) {
    __shared__ u64 warp_max[8];
    __shared__ double warp_sum[8];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int64_t row = blockIdx.x;
    const T* xr = x + row * ldx;

    u64 mx = 0;
    double sum = 0.0;
    for (int64_t chunk = warp; chunk < chunks; chunk += 8) {
        float f[8];
        load8<T>(xr, chunk * 256 + lane * 8, D, vec_ok != 0, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const u64 a = uabs(decimal_round(f[e], dec_scale, dec_mult));
            mx = a > mx ? a : mx;
            if (clip_k > 0.0f) sum += static_cast<double>(a);
        }
    }
    mx = warp_max_u64(mx);
    if (clip_k > 0.0f) sum = warp_sum_f64(sum);
    if (lane == 0) {
        warp_max[warp] = mx;
        warp_sum[warp] = sum;
    }
    __syncthreads();
    mx = warp_max[0];
    sum = warp_sum[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        mx = warp_max[i] > mx ? warp_max[i] : mx;
        sum += warp_sum[i];
    }
    const int shift = clip_k > 0.0f ? shift_for_clipped(mx, sum, static_cast<int>(D), bits, clip_k) : shift_for(mx, bits);
    if (threadIdx.x == 0) {
        if (scales != nullptr) scales[row] = static_cast<float>(1ull << shift);
        if (shifts != nullptr) shifts[row] = shift;
    }
    for (int64_t chunk = warp; chunk < chunks; chunk += 8) {
        float f[8];
        load8<T>(xr, chunk * 256 + lane * 8, D, vec_ok != 0, f);
        long long v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = decimal_round(f[e], dec_scale, dec_mult);
        emit_chunk(v, shift, bits, lane, chunk, W,
                   words != nullptr ? words + row * bits * W : nullptr,
                   q8 != nullptr ? q8 + row * ld8 : nullptr);
    }
}

// What a dot's exactness test needs of one 256-element chunk of keys: the sum of |k| over the warp's bytes; the lane's
// part of the sum of k^2 is added to lane_sq.
__device__ __forceinline__ void chunk_sums(u64 packed, int& abs_sum, int& lane_sq) {
    const uint32_t lo = static_cast<uint32_t>(packed), hi = static_cast<uint32_t>(packed >> 32);
    // +-1 per byte by its sign: k * sign(k) = |k|
    const int slo = static_cast<int>(prmt(lo, lo, 0xba98u) | 0x01010101u), shi = static_cast<int>(prmt(hi, hi, 0xba98u) | 0x01010101u);
    const int a = __dp4a(static_cast<int>(hi), shi, __dp4a(static_cast<int>(lo), slo, 0));
    lane_sq = __dp4a(static_cast<int>(hi), static_cast<int>(hi), __dp4a(static_cast<int>(lo), static_cast<int>(lo), lane_sq));
    abs_sum = __reduce_add_sync(0xffffffffu, a);
}

// One chunk of a row on the 64-bit path with the row's shift; returns the lane's bytes.
template <typename T>
__device__ __noinline__ u64 generic_row_chunk(const T* xr, int64_t chunk, int64_t D, double dec_scale, uint32_t dec_mult,
                                              int bits, int vec_ok, int lane, int shift) {
    float f[8];
    load8<T>(xr, chunk * 256 + lane * 8, D, vec_ok != 0, f);
    long long v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = decimal_round(f[e], dec_scale, dec_mult);
    return quantise8(v, shift, bits);
}

// The shift of a row on the 64-bit path, found by one warp.
template <typename T>
__device__ __noinline__ int generic_row_shift(const T* xr, int64_t chunks, int64_t D, double dec_scale, uint32_t dec_mult,
                                              int bits, int vec_ok, int lane) {
    u64 mx = 0;
    for (int64_t chunk = 0; chunk < chunks; ++chunk) {
        float f[8];
        load8<T>(xr, chunk * 256 + lane * 8, D, vec_ok != 0, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const u64 a = uabs(decimal_round(f[e], dec_scale, dec_mult));
            mx = a > mx ? a : mx;
        }
    }
    return shift_for(warp_max_u64(mx), bits);
}

// Row mode (keys) with the row kept in registers: x is read once. 2^wpr_log2 warps share a row, CPW chunks each, and
// a block of 8 warps takes 8 >> wpr_log2 rows; the row's largest |x| goes through shared memory once, and because
// rounding is monotonic its bit pattern alone gives the shift. The bytes go to the int8 image and, traded among four
// lanes, to the slices; the same pass leaves the slice weights and the row's bounds (sum of |k|, largest such sum
// over a chunk, sum of k^2), which took ten library kernels over 32-bit copies of the image before.
// Bound by HBM: 4 bytes in and 1 + bits / 8 out per element (float32). A row with NaN, inf or |x * 10^dp| beyond the
// fast range is redone from memory on the 64-bit path, every warp finding the shift for itself.
template <typename T, int CPW>
__global__ void __launch_bounds__(256, CPW * RawLane<T>::kVecs <= 8 ? 4 : 2) quantize_pack_row_fast_kernel(
    const T* __restrict__ x, int64_t rows, int64_t D, int64_t ldx, double dec_scale, uint32_t dec_mult, int bits,
    int chunks, int64_t W, int wpr_log2, u64* __restrict__ words, float* __restrict__ scales,
    int32_t* __restrict__ shifts, int8_t* __restrict__ q8, int64_t ld8, int vec_ok, float* __restrict__ slice_weights,
    float* __restrict__ bounds) {
    __shared__ uint32_t wmax[8];
    __shared__ int wsum[3][8];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wpr = 1 << wpr_log2;
    const int sub = warp & (wpr - 1);
    const int64_t row = static_cast<int64_t>(blockIdx.x) * (8 >> wpr_log2) + (warp >> wpr_log2);
    const bool row_ok = row < rows;
    const T* xr = x + (row_ok ? row : 0) * ldx;

    RawLane<T> raw[CPW];
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
        const int64_t col = static_cast<int64_t>(sub + i * wpr) * 256 + lane * 8;
        const int64_t left = row_ok ? D - col : 0;
        if (vec_ok && left >= 8) raw[i].load(xr + col);
        else raw[i].load_tail(xr + (left > 0 ? col : 0), left);
    }
    uint32_t amax_bits = 0;
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
        if constexpr (sizeof(T) == 4) amax_bits = max(amax_bits, raw[i].abs_max_masked());
        else amax_bits = max(amax_bits, raw[i].abs_max());
    }
    amax_bits = __reduce_max_sync(0xffffffffu, amax_bits);
    if (lane == 0) wmax[warp] = amax_bits;
    __syncthreads();
    const int group = warp & ~(wpr - 1);
    for (int i = 0; i < wpr; ++i) amax_bits = max(amax_bits, wmax[group + i]);
    const float mult = static_cast<float>(dec_mult);
    int shift = fast_group_shift(RawLane<T>::abs_value(amax_bits), mult, bits);
    const bool fast = shift >= 0;
    const bool clamp = fast && needs_clamp(RawLane<T>::abs_value(amax_bits), mult, shift, bits);
    if (!fast) shift = generic_row_shift<T>(xr, chunks, D, dec_scale, dec_mult, bits, vec_ok, lane);

    int asum = 0, amax_chunk = 0, qsum = 0;
    const int s0 = first_slice(lane);
    int8_t* q8_out = q8 + row * ld8 + sub * 256 + lane * 8;
    // half word (lane / 4) % 2 of the lane's word in slice s0, and in the slice after it
    uint32_t* w_out = reinterpret_cast<uint32_t*>(words + (row * bits + s0) * W + sub * 4 + (lane >> 3)) + ((lane >> 2) & 1);
    uint32_t* w_out1 = w_out + 2 * W;
    const int words_left = static_cast<int>(W) - sub * 4 - (lane >> 3);      // the lane's word exists while this is positive
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
        const int chunk = sub + i * wpr;
        if (row_ok && chunk < chunks) {
            u64 packed;
            if (fast) {
                packed = clamp ? raw[i].template quantise<true>(mult, shift, bits) : raw[i].template quantise<false>(mult, shift, bits);
            } else {
                packed = generic_row_chunk<T>(xr, chunk, D, dec_scale, dec_mult, bits, vec_ok, lane, shift);
            }
            if (q8 != nullptr) *reinterpret_cast<u64*>(q8_out + i * wpr * 256) = packed;
            if (words != nullptr) {
                uint32_t w0, w1;
                slice_pieces(packed, lane, w0, w1);
                if (words_left > i * wpr * 4) {
                    if (s0 < bits) w_out[i * wpr * 8] = w0;
                    if (s0 + 1 < bits) w_out1[i * wpr * 8] = w1;
                }
            }
            if (bounds != nullptr) {
                int a;
                chunk_sums(packed, a, qsum);
                asum += a;
                amax_chunk = max(amax_chunk, a);
            }
        }
    }
    if (bounds != nullptr) qsum = __reduce_add_sync(0xffffffffu, qsum);
    const float scale = static_cast<float>(1ull << shift);
    if (row_ok && sub == 0) {
        if (lane == 0) {
            if (scales != nullptr) scales[row] = scale;
            if (shifts != nullptr) shifts[row] = shift;
        }
        if (slice_weights != nullptr && lane < bits) slice_weights[row * bits + lane] = slice_weight(lane, bits, scale);
    }
    if (bounds != nullptr) {
        if (lane == 0) {
            wsum[0][warp] = asum;
            wsum[1][warp] = amax_chunk;
            wsum[2][warp] = qsum;
        }
        __syncthreads();
        if (row_ok && sub == 0 && lane == 0) {
            for (int i = 1; i < wpr; ++i) {
                asum += wsum[0][warp + i];
                amax_chunk = max(amax_chunk, wsum[1][warp + i]);
                qsum += wsum[2][warp + i];
            }
            bounds[row] = static_cast<float>(asum);
            bounds[rows + row] = static_cast<float>(amax_chunk);
            bounds[2 * rows + row] = static_cast<float>(qsum);
        }
    }
}

// The same for what a key build asks for, every output. The kernel above was bound by instruction issue (266 a chunk of 256
// elements, 77 % of the slots), so nothing is decided per chunk here that is known before: WPR warps on a row and CPW chunks each
// are constants (all addresses a base and an immediate), the clamp and the 64-bit path are chosen once per row, and the outputs are
// there. The largest magnitude comes from signed and unsigned maxima of the patterns, three at a time, without masking each. 174
// instructions a chunk, 16384 x 4096 float32: 82.8 -> 64.3 us (385 MB, 93 % of the copy rate), 50000 x 768 57.7 -> 40.1.
// kWhole: rows of whole chunks on 16-byte vectors; else the last chunk's lanes look at what is left.
template <typename T, int CPW, int WPR, bool kWhole>
__global__ void __launch_bounds__(256, CPW * RawLane<T>::kVecs <= 8 ? 4 : 2) quantize_pack_row_build_kernel(
    const T* __restrict__ x, uint32_t rows, int64_t D, uint32_t ldx, int vec_ok, double dec_scale, uint32_t dec_mult, int bits, int chunks, uint32_t W,
    u64* __restrict__ words, float* __restrict__ scales, int32_t* __restrict__ shifts, int8_t* __restrict__ q8, uint32_t ld8,
    float* __restrict__ slice_weights, float* __restrict__ bounds) {
    __shared__ uint32_t wmax[8];
    __shared__ int wsum[3][8];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int sub = warp & (WPR - 1);
    const uint32_t row = blockIdx.x * (8u / WPR) + static_cast<uint32_t>(warp / WPR);
    const bool row_ok = row < rows;
    const int mine = row_ok ? (chunks - sub + WPR - 1) / WPR : 0;        // chunks sub, sub + WPR, .. of the row
    const T* xr = x + static_cast<size_t>(row_ok ? row : 0u) * ldx;
    const T* src = xr + sub * 256 + lane * 8;

    RawLane<T> raw[CPW];
#pragma unroll
    for (int i = 0; i < CPW; ++i) {
        if (kWhole && i < mine) {
            raw[i].load(src + i * WPR * 256);
        } else if (!kWhole && i < mine) {
            const int64_t left = D - (sub + i * WPR) * 256 - lane * 8;
            if (vec_ok && left >= 8) raw[i].load(src + i * WPR * 256);
            else raw[i].load_tail(left > 0 ? src + i * WPR * 256 : xr, left);
        } else {
#pragma unroll
            for (int e = 0; e < RawLane<T>::kVecs; ++e) raw[i].v[e] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    uint32_t amax_bits = 0;
    if constexpr (sizeof(T) == 4) {
        int positive = 0;           // positive patterns order as signed, negative ones above them as unsigned numbers
        uint32_t negative = 0;
#pragma unroll
        for (int i = 0; i < CPW; ++i) {
#pragma unroll
            for (int e = 0; e < RawLane<T>::kVecs; ++e) {
                const uint4& a = raw[i].v[e];
                positive = __vimax3_s32(__vimax3_s32(positive, static_cast<int>(a.x), static_cast<int>(a.y)), static_cast<int>(a.z), static_cast<int>(a.w));
                negative = __vimax3_u32(__vimax3_u32(negative, a.x, a.y), a.z, a.w);
            }
        }
        amax_bits = max(static_cast<uint32_t>(positive), (negative >> 31) != 0u ? negative & 0x7fffffffu : 0u);
    } else {
#pragma unroll
        for (int i = 0; i < CPW; ++i) amax_bits = max(amax_bits, raw[i].abs_max());
    }
    amax_bits = __reduce_max_sync(0xffffffffu, amax_bits);
    if constexpr (WPR > 1) {
        if (lane == 0) wmax[warp] = amax_bits;
        __syncthreads();
        const int group = warp & ~(WPR - 1);
#pragma unroll
        for (int i = 0; i < WPR; ++i) amax_bits = max(amax_bits, wmax[group + i]);
    }
    const float mult = static_cast<float>(dec_mult);
    int shift = fast_group_shift(RawLane<T>::abs_value(amax_bits), mult, bits);
    const bool fast = shift >= 0;
    const bool clamp = fast && needs_clamp(RawLane<T>::abs_value(amax_bits), mult, shift, bits);
    if (!fast) shift = generic_row_shift<T>(xr, chunks, D, dec_scale, dec_mult, bits, vec_ok, lane);

    int asum = 0, amax_chunk = 0, qsum = 0;
    const int s0 = first_slice(lane);
    const bool first_there = s0 < bits, second_there = s0 + 1 < bits;
    int8_t* q8_out = q8 + static_cast<size_t>(row_ok ? row : 0u) * ld8 + sub * 256 + lane * 8;
    // half word (lane / 4) % 2 of the lane's word in slice s0, and in the slice after it
    uint32_t* w_out = reinterpret_cast<uint32_t*>(words + (static_cast<size_t>(row_ok ? row : 0u) * bits + s0) * W + sub * 4 + (lane >> 3)) + ((lane >> 2) & 1);
    uint32_t* w_out1 = w_out + 2u * W;
    const int words_left = static_cast<int>(W) - sub * 4 - (lane >> 3);      // the lane's word exists while this is positive
    auto emit = [&](u64 packed, int i) {
        *reinterpret_cast<u64*>(q8_out + i * WPR * 256) = packed;
        uint32_t w0, w1;
        slice_pieces(packed, lane, w0, w1);
        if (kWhole || words_left > i * WPR * 4) {
            if (first_there) w_out[i * WPR * 8] = w0;
            if (second_there) w_out1[i * WPR * 8] = w1;
        }
        int a;
        chunk_sums(packed, a, qsum);
        asum += a;
        amax_chunk = max(amax_chunk, a);
    };
    if (fast && !clamp) {
#pragma unroll
        for (int i = 0; i < CPW; ++i)
            if (i < mine) emit(raw[i].template quantise<false>(mult, shift, bits), i);
    } else if (fast) {
#pragma unroll
        for (int i = 0; i < CPW; ++i)
            if (i < mine) emit(raw[i].template quantise<true>(mult, shift, bits), i);
    } else {
#pragma unroll 1
        for (int i = 0; i < mine; ++i)
            emit(generic_row_chunk<T>(xr, sub + i * WPR, D, dec_scale, dec_mult, bits, vec_ok, lane, shift), i);
    }
    qsum = __reduce_add_sync(0xffffffffu, qsum);
    const float scale = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);      // 2^shift, shift <= 62
    if (row_ok && sub == 0) {
        if (lane == 0) {
            scales[row] = scale;
            if (shifts != nullptr) shifts[row] = shift;
        }
        if (lane < bits) slice_weights[static_cast<size_t>(row) * bits + lane] = slice_weight(lane, bits, scale);
    }
    if constexpr (WPR > 1) {
        if (lane == 0) {
            wsum[0][warp] = asum;
            wsum[1][warp] = amax_chunk;
            wsum[2][warp] = qsum;
        }
        __syncthreads();
    }
    if (row_ok && sub == 0 && lane == 0) {
#pragma unroll
        for (int i = 1; i < WPR; ++i) {
            asum += wsum[0][warp + i];
            amax_chunk = max(amax_chunk, wsum[1][warp + i]);
            qsum += wsum[2][warp + i];
        }
        bounds[row] = static_cast<float>(asum);
        bounds[static_cast<size_t>(rows) + row] = static_cast<float>(amax_chunk);
        bounds[2 * static_cast<size_t>(rows) + row] = static_cast<float>(qsum);
    }
}

// Bounds of an int8 image that exists already (loaded key sets, rows too long for the kernel above): one warp per row.
__global__ void __launch_bounds__(256) key_bounds_kernel(const int8_t* __restrict__ q8, int64_t rows, int64_t chunks,
                                                         int64_t ld8, float* __restrict__ bounds) {
    const int lane = threadIdx.x & 31;
    const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const u64* src = reinterpret_cast<const u64*>(q8 + row * ld8) + lane;
    long long asum = 0, qsum = 0;
    int amax_chunk = 0;
#pragma unroll 4
    for (int64_t c = 0; c < chunks; ++c) {
        int a, q = 0;
        chunk_sums(__ldg(src + c * 32), a, q);
        asum += a;
        qsum += __reduce_add_sync(0xffffffffu, q);
        amax_chunk = max(amax_chunk, a);
    }
    if (lane == 0) {
        bounds[row] = static_cast<float>(asum);
        bounds[rows + row] = static_cast<float>(amax_chunk);
        bounds[2 * rows + row] = static_cast<float>(qsum);
    }
}

// Slice weights behind the generic kernels; scales: one per row, or null for chunk mode.
__global__ void __launch_bounds__(256) slice_weights_kernel(const float* __restrict__ scales, int64_t n, int bits,
                                                            float* __restrict__ slice_weights) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
    if (i >= n) return;
    const int64_t row = i / bits;
    slice_weights[i] = slice_weight(static_cast<int>(i - row * bits), bits, scales != nullptr ? scales[row] : 1.0f);
}

__global__ void __launch_bounds__(256) recombine_i8_kernel(
    const u64* __restrict__ words, int64_t rows, int bits, int64_t W, int64_t chunks,
    int8_t* __restrict__ q8, int64_t ld8) {
    const int lane = threadIdx.x & 31;
    const int64_t unit = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (unit >= rows * chunks) return;
    const int64_t row = unit / chunks;
    const int64_t chunk = unit - row * chunks;
    const int64_t word = chunk * 4 + (lane >> 3);
    u64 t = 0;
    if (word < W) {
        const uint8_t* src = reinterpret_cast<const uint8_t*>(words + row * bits * W + word) + (lane & 7);
        for (int s = 0; s < bits; ++s) {
            t |= static_cast<u64>(src[static_cast<size_t>(s) * static_cast<size_t>(W) * 8u]) << (8 * s);
        }
    }
    u64 vals = transpose8x8(t);  // byte e = the `bits`-bit two's-complement value of element e
    // Sign-extend each byte from `bits` bits: where bit (bits-1) is set, set the bits above it.
    // sign holds 0 or 1 per byte and fill < 256, so the product never carries across bytes.
    const u64 sign = (vals >> (bits - 1)) & 0x0101010101010101ull;
    const u64 fill = (0xffull << bits) & 0xffull;
    vals |= sign * fill;
    *reinterpret_cast<u64*>(q8 + row * ld8 + chunk * 256 + lane * 8) = vals;
}

template <typename Y>
__device__ __forceinline__ Y from_float(float v);
template <>
__device__ __forceinline__ float from_float<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// y = cast(out) + cast(bias), the add evaluated in float on the two already-narrowed values and
// narrowed again, which is what the reference's `scores.to(dtype) + bias.to(dtype)` does.
template <typename Y>
__global__ void __launch_bounds__(256) cast_bias_kernel(const float* __restrict__ out, int64_t ldo,
                                                        const float* __restrict__ bias, int64_t Q,
                                                        int64_t R, Y* __restrict__ y, int64_t ldy) {
    const int64_t per_row = (R + 3) / 4;
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= Q * per_row) return;
    const int64_t q = idx / per_row;
    const int64_t r0 = (idx - q * per_row) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int64_t r = r0 + e;
        if (r < R) {
            const Y narrowed = from_float<Y>(out[q * ldo + r]);
            if (bias != nullptr) {
                const Y b = from_float<Y>(bias[r]);
                y[q * ldy + r] = from_float<Y>(to_float(narrowed) + to_float(b));
            } else {
                y[q * ldy + r] = narrowed;
            }
        }
    }
}

}  // namespace
}  // namespace bsi

namespace bsi {
namespace {
// Blocks of 256 threads of `kernel` that fit the current device at once (cached per kernel).
template <auto kernel>
int64_t resident_blocks() {
    static thread_local int cached_dev = -1;
    static thread_local int cached = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) { set_error("quantize_pack: cudaGetDevice failed"); return -1; }
    if (dev != cached_dev) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess || per_sm <= 0) {
            set_error("quantize_pack: occupancy query failed");
            return -1;
        }
        cached = per_sm * sm_count();
        cached_dev = dev;
    }
    return cached;
}
struct PackArgs {
    int64_t rows, D, ldx, ld8, chunks, W;
    double dec_scale;
    uint32_t dec_mult;
    int bits;
    u64* words;
    float* scales;
    int32_t* shifts;
    int8_t* q8;
    int vec_ok;
    cudaStream_t stream;
    float clip_k;
    float* sq_norms;
    float* slice_weights;
    float* key_bounds;    // row mode only
};

// Turns per warp: four, two or one, as many as leave a block for every place on the chip and few lanes without a unit (a row's
// last warp and, for an odd number of chunks, its last turn are not full: 2500 x 2304 with four turns 7.6 us, pair kernel 6.5).
// Below that the other kernels spread the units better.
template <typename T, bool kWords>
int launch_chunk_turns(const T* x, const PackArgs& a, bool* taken) {
    *taken = false;
    const int64_t turns = (a.chunks + 1) / 2, places = static_cast<int64_t>(sm_count()) * 4;
    int g = 4;
    auto fits = [&] {
        const int64_t warps = (turns + g - 1) / g;
        return (a.rows * warps + 7) / 8 >= places && warps * g * 2 * 8 <= a.chunks * 9;
    };
    while (g > 1 && !fits()) g /= 2;
    if (!fits()) return BSI_OK;
    const int64_t per_row = (turns + g - 1) / g, blocks = (a.rows * per_row + 7) / 8;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(blocks), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = a.stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    auto kernel = g == 4 ? quantize_pack_chunk_turns_kernel<T, 4, kWords>
                         : g == 2 ? quantize_pack_chunk_turns_kernel<T, 2, kWords> : quantize_pack_chunk_turns_kernel<T, 1, kWords>;
    BSI_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, x, static_cast<uint32_t>(a.rows), static_cast<uint32_t>(per_row), static_cast<uint32_t>(a.chunks),
                                    a.dec_scale, a.dec_mult, a.bits, a.words, a.scales, a.q8, a.sq_norms, a.slice_weights));
    *taken = true;
    return BSI_OK;
}

template <typename T, bool kDense, bool kWords, bool kQ8>
int launch_chunk_fast(const T* x, const PackArgs& a) {
    // one unit per warp and turn while a turn takes them all, else two (16-bit types)
    auto kernel = quantize_pack_chunk_fast_kernel<T, kDense, kWords, kQ8>;
    int64_t resident = resident_blocks<quantize_pack_chunk_fast_kernel<T, kDense, kWords, kQ8>>();
    if (resident <= 0) return BSI_ERR_CUDA;
    int64_t blocks = (a.rows * a.chunks + 7) / 8;
    if constexpr (sizeof(T) == 2) {
        if (blocks > resident) {
            kernel = quantize_pack_chunk_pair_kernel<T, kDense, kWords, kQ8>;
            resident = resident_blocks<quantize_pack_chunk_pair_kernel<T, kDense, kWords, kQ8>>();
            if (resident <= 0) return BSI_ERR_CUDA;
            blocks = (a.rows * a.chunks + 15) / 16;
        }
    }
    blocks = blocks < resident ? blocks : resident;
    FastGeom g;
    g.total = static_cast<uint32_t>(a.rows * a.chunks);
    g.chunks = static_cast<uint32_t>(a.chunks);
    g.D = static_cast<uint32_t>(a.D);
    g.ldx = static_cast<uint32_t>(a.ldx);
    g.ld8 = static_cast<uint32_t>(kQ8 ? a.ld8 : 0);
    g.W = static_cast<uint32_t>(a.W);
    g.row_bytes = static_cast<uint32_t>(a.bits * a.W * 8);
    g.slice_bytes = static_cast<uint32_t>(a.W * 8);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(static_cast<unsigned>(blocks), 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.stream = a.stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    BSI_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, x, g, a.dec_scale, a.dec_mult,
                                    a.bits, a.words, a.scales, a.shifts, a.q8, a.vec_ok, a.sq_norms, a.slice_weights));
    return BSI_OK;
}

int launch_slice_weights(const float* scales, const PackArgs& a) {
    if (a.slice_weights == nullptr) return BSI_OK;
    const int64_t n = a.rows * a.bits;
    slice_weights_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, a.stream>>>(scales, n, a.bits, a.slice_weights);
    return BSI_OK;
}

template <typename T, int CPW, int WPR, bool kWhole>
int launch_row_build(const T* x, const PackArgs& a, unsigned grid) {
    quantize_pack_row_build_kernel<T, CPW, WPR, kWhole><<<grid, 256, 0, a.stream>>>(
        x, static_cast<uint32_t>(a.rows), a.D, static_cast<uint32_t>(a.ldx), a.vec_ok, a.dec_scale, a.dec_mult, a.bits,
        static_cast<int>(a.chunks), static_cast<uint32_t>(a.W), a.words, a.scales, a.shifts, a.q8, static_cast<uint32_t>(a.ld8),
        a.slice_weights, a.key_bounds);
    return BSI_OK;
}

// Row mode: the register-resident kernel for rows of up to 64 chunks (8 warps x 8 chunks), decimal_places in [0, 8]
// and no clipping; the two-pass 64-bit kernel otherwise. As few warps on a row (1, 2, 4 or 8) as leave each four chunks at
// most, more than that only on the longest rows: what a row costs beside its chunks is paid per warp (16384 x 4096
// float32, an earlier form: 96 us with 8 warps of 2 chunks, 84 us with 4 of 4; 4096 x 768: 9.2 us with 4 warps of 1, 7.2 us with 2 of 2).
template <typename T>
int launch_row(const T* x, const PackArgs& a) {
    if (a.dec_mult == 0u || a.clip_k > 0.0f || a.chunks > 64) {
        quantize_pack_row_kernel<T><<<static_cast<unsigned>(a.rows), 256, 0, a.stream>>>(
            x, a.rows, a.D, a.ldx, a.dec_scale, a.dec_mult, a.bits, a.chunks, a.W, a.words, a.scales, a.shifts, a.q8, a.ld8,
            a.vec_ok, a.clip_k);
        if (a.slice_weights != nullptr && a.scales == nullptr)
            return fail(BSI_ERR_INVALID, "quantize_pack: row-mode slice weights need the scales as well");
        if (int rc = launch_slice_weights(a.scales, a)) return rc;
        if (a.key_bounds != nullptr) {
            if (a.q8 == nullptr) return fail(BSI_ERR_INVALID, "quantize_pack: key bounds need the int8 image as well");
            key_bounds_kernel<<<static_cast<unsigned>((a.rows + 7) / 8), 256, 0, a.stream>>>(a.q8, a.rows, a.chunks, a.ld8,
                                                                                          a.key_bounds);
        }
        return BSI_OK;
    }
    int wpr_log2 = 0;
    while (wpr_log2 < 3 && ((a.chunks + (1 << wpr_log2) - 1) >> wpr_log2) > 4) ++wpr_log2;
    const int64_t per_block = 8 >> wpr_log2;
    const unsigned grid = static_cast<unsigned>((a.rows + per_block - 1) / per_block);
    const int cpw = static_cast<int>((a.chunks + (1 << wpr_log2) - 1) >> wpr_log2);
    if (a.words != nullptr && a.q8 != nullptr && a.scales != nullptr && a.slice_weights != nullptr && a.key_bounds != nullptr &&
        a.rows < (1ll << 31) && a.ldx < (1ll << 31) && a.ld8 < (1ll << 31)) {
        const bool whole = a.vec_ok && a.D == a.chunks * 256;
#define BSI_ROW_BUILD(CPW, WPR) (whole ? launch_row_build<T, CPW, WPR, true>(x, a, grid) : launch_row_build<T, CPW, WPR, false>(x, a, grid))
        if (wpr_log2 == 0) return cpw <= 1 ? BSI_ROW_BUILD(1, 1) : cpw <= 2 ? BSI_ROW_BUILD(2, 1) : BSI_ROW_BUILD(4, 1);
        if (wpr_log2 == 1) return BSI_ROW_BUILD(4, 2);
        if (wpr_log2 == 2) return BSI_ROW_BUILD(4, 4);
        return cpw <= 4 ? BSI_ROW_BUILD(4, 8) : BSI_ROW_BUILD(8, 8);
#undef BSI_ROW_BUILD
    }
#define BSI_ROW_FAST(CPW)                                                                                              \
    quantize_pack_row_fast_kernel<T, CPW><<<grid, 256, 0, a.stream>>>(                                                 \
        x, a.rows, a.D, a.ldx, a.dec_scale, a.dec_mult, a.bits, static_cast<int>(a.chunks), a.W, wpr_log2, a.words,    \
        a.scales, a.shifts, a.q8, a.ld8, a.vec_ok, a.slice_weights, a.key_bounds)
    if (cpw <= 1) BSI_ROW_FAST(1);
    else if (cpw <= 2) BSI_ROW_FAST(2);
    else if (cpw <= 4) BSI_ROW_FAST(4);
    else BSI_ROW_FAST(8);
#undef BSI_ROW_FAST
    return BSI_OK;
}

// Chunk mode: the fast kernel when its preconditions hold (decimal_places in [0, 8], scales
// wanted, every offset below 2^31, no outlier clipping), else the generic kernel.
template <typename T>
int launch_chunk(const T* x, const PackArgs& a) {
    int64_t widest = a.chunks * 256;
    if (a.ldx > widest) widest = a.ldx;
    if (a.q8 != nullptr && a.ld8 > widest) widest = a.ld8;
    const bool fast = a.dec_mult != 0u && a.scales != nullptr && !(a.clip_k > 0.0f) &&
                      a.rows * widest < (1ll << 31) && (a.words != nullptr || a.q8 != nullptr);
    if (!fast) {
        int64_t blocks = (a.rows * a.chunks + 7) / 8;
        const int64_t cap = static_cast<int64_t>(sm_count()) * 64;
        blocks = blocks < cap ? blocks : cap;
        quantize_pack_chunk_generic_kernel<T><<<static_cast<unsigned>(blocks), 256, 0, a.stream>>>(
            x, a.rows, a.D, a.ldx, a.dec_scale, a.dec_mult, a.bits, a.chunks, a.W, a.words, a.scales, a.shifts, a.q8,
            a.ld8, a.vec_ok, a.clip_k, a.sq_norms);
        return launch_slice_weights(nullptr, a);
    }
    const bool dense = a.vec_ok && a.ldx == a.D && (a.D & 255) == 0 && (a.q8 == nullptr || a.ld8 == a.D);
    const bool w = a.words != nullptr, q = a.q8 != nullptr;
    if constexpr (sizeof(T) == 2) {
        if (dense && q && a.sq_norms != nullptr && a.shifts == nullptr && w == (a.slice_weights != nullptr)) {
            bool taken = false;
            const int rc = w ? launch_chunk_turns<T, true>(x, a, &taken) : launch_chunk_turns<T, false>(x, a, &taken);
            if (rc != BSI_OK || taken) return rc;
        }
    }
    if (dense) {
        if (w && q) return launch_chunk_fast<T, true, true, true>(x, a);
        if (q) return launch_chunk_fast<T, true, false, true>(x, a);
        return launch_chunk_fast<T, true, true, false>(x, a);
    }
    if (w && q) return launch_chunk_fast<T, false, true, true>(x, a);
    if (q) return launch_chunk_fast<T, false, false, true>(x, a);
    return launch_chunk_fast<T, false, true, false>(x, a);
}
}  // namespace
}  // namespace bsi

extern "C" int bsi_b200_quantize_pack(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx,
                                      int decimal_places, int bits, int chunk_mode,
                                      uint64_t* words, float* scales, int32_t* shifts,
                                      int8_t* q8, int64_t ld8, bsi_stream_t stream_) {
    return bsi_b200_quantize_pack_clip(x, dtype, rows, D, ldx, decimal_places, bits, chunk_mode, 0.0f, words, scales,
                                       shifts, q8, ld8, stream_);
}

extern "C" int bsi_b200_quantize_pack_clip(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx,
                                           int decimal_places, int bits, int chunk_mode, float clip_k,
                                           uint64_t* words, float* scales, int32_t* shifts,
                                           int8_t* q8, int64_t ld8, bsi_stream_t stream_) {
    return bsi_b200_quantize_pack_norms(x, dtype, rows, D, ldx, decimal_places, bits, chunk_mode, clip_k, words, scales,
                                        shifts, q8, ld8, nullptr, stream_);
}

extern "C" int bsi_b200_quantize_pack_norms(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx,
                                            int decimal_places, int bits, int chunk_mode, float clip_k,
                                            uint64_t* words, float* scales, int32_t* shifts,
                                            int8_t* q8, int64_t ld8, float* sq_norms, bsi_stream_t stream_) {
    return bsi_b200_quantize_pack_all(x, dtype, rows, D, ldx, decimal_places, bits, chunk_mode, clip_k, words, scales,
                                      shifts, q8, ld8, sq_norms, nullptr, nullptr, stream_);
}

extern "C" int bsi_b200_quantize_pack_all(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx,
                                          int decimal_places, int bits, int chunk_mode, float clip_k,
                                          uint64_t* words, float* scales, int32_t* shifts,
                                          int8_t* q8, int64_t ld8, float* sq_norms, float* slice_weights,
                                          float* key_bounds, bsi_stream_t stream_) {
    using namespace bsi;
    if (key_bounds != nullptr && chunk_mode)
        return fail(BSI_ERR_UNSUPPORTED, "quantize_pack: key bounds are per row: row mode only");
    if (sq_norms != nullptr && !chunk_mode)
        return fail(BSI_ERR_UNSUPPORTED, "quantize_pack: sums of squares are per (row, chunk): chunk mode only");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (rows < 0 || D < 0 || ldx < D) return fail(BSI_ERR_INVALID, "quantize_pack: bad rows/D/ldx");
    if (bits < 2 || bits > 8) return fail(BSI_ERR_UNSUPPORTED, "quantize_pack: bits must be in [2, 8]");
    if (dtype != BSI_DTYPE_F32 && dtype != BSI_DTYPE_F16 && dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_INVALID, "quantize_pack: unknown dtype");
    if (rows == 0 || D == 0) return BSI_OK;
    if (x == nullptr) return fail(BSI_ERR_INVALID, "quantize_pack: x is null");
    const int64_t chunks = (D + 255) / 256;
    const int64_t W = (D + 63) / 64;
    if (q8 != nullptr) {
        if (ld8 < chunks * 256 || (ld8 & 15) != 0 || (reinterpret_cast<uintptr_t>(q8) & 15) != 0)
            return fail(BSI_ERR_INVALID, "quantize_pack: q8 needs ld8 >= 256*ceil(D/256), ld8 % 16 == 0, 16-byte base");
    }
    if (int rc = require_sm100()) return rc;
    const int esz = dtype == BSI_DTYPE_F32 ? 4 : 2;
    const int vec_ok = ((reinterpret_cast<uintptr_t>(x) & 15) == 0 && ((ldx * esz) & 15) == 0) ? 1 : 0;
    const double dec_scale = pow(10.0, static_cast<double>(decimal_places));
    uint32_t dec_mult = 0;  // 10^dp when it is a small integer; 0 = use the float64 expression
    if (decimal_places >= 0 && decimal_places <= 8) {
        dec_mult = 1;
        for (int i = 0; i < decimal_places; ++i) dec_mult *= 10u;
    }
    u64* w = reinterpret_cast<u64*>(words);

    if (!chunk_mode && rows > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "quantize_pack: too many rows for one launch");
    const PackArgs a{rows, D, ldx, ld8, chunks, W, dec_scale, dec_mult, bits, w, scales, shifts, q8, vec_ok, stream, clip_k,
                     sq_norms, slice_weights, key_bounds};
    int rc;
    if (dtype == BSI_DTYPE_F32)
        rc = chunk_mode ? launch_chunk<float>(static_cast<const float*>(x), a) : launch_row<float>(static_cast<const float*>(x), a);
    else if (dtype == BSI_DTYPE_F16)
        rc = chunk_mode ? launch_chunk<__half>(static_cast<const __half*>(x), a) : launch_row<__half>(static_cast<const __half*>(x), a);
    else
        rc = chunk_mode ? launch_chunk<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(x), a)
                        : launch_row<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(x), a);
    if (rc != BSI_OK) return rc;
    return check_launch("quantize_pack launch");
}

extern "C" int bsi_b200_quantize_pack_multi(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx,
                                            int decimal_places, int bits, int n_q8_dst, int8_t* const* q8_dst,
                                            int64_t ld8, int n_scale_dst, float* const* scale_dst, int64_t scale_ld,
                                            bsi_stream_t stream_) {
    using namespace bsi;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (rows < 0 || D < 0 || ldx < D) return fail(BSI_ERR_INVALID, "quantize_pack_multi: bad rows/D/ldx");
    if (bits < 2 || bits > 8) return fail(BSI_ERR_UNSUPPORTED, "quantize_pack_multi: bits must be in [2, 8]");
    if (dtype != BSI_DTYPE_F32 && dtype != BSI_DTYPE_F16 && dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_INVALID, "quantize_pack_multi: unknown dtype");
    if (n_q8_dst < 1 || n_q8_dst > BSI_B200_MAX_PEERS || n_scale_dst < 1 || n_scale_dst > BSI_B200_MAX_PEERS ||
        q8_dst == nullptr || scale_dst == nullptr)
        return fail(BSI_ERR_INVALID, "quantize_pack_multi: bad destinations");
    if (rows == 0 || D == 0) return BSI_OK;
    if (x == nullptr) return fail(BSI_ERR_INVALID, "quantize_pack_multi: x is null");
    if ((D & 255) != 0) return fail(BSI_ERR_UNSUPPORTED, "quantize_pack_multi: D must be a multiple of 256");
    const int64_t chunks = D / 256;
    const int esz = dtype == BSI_DTYPE_F32 ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(x) & 15) != 0 || ((ldx * esz) & 15) != 0)
        return fail(BSI_ERR_INVALID, "quantize_pack_multi: x needs 16-byte aligned rows");
    if (ld8 < D || (ld8 & 7) != 0 || scale_ld < chunks)
        return fail(BSI_ERR_INVALID, "quantize_pack_multi: ld8 >= D, ld8 % 8 == 0 and scale_ld >= D/256 are required");
    int64_t widest = ldx > ld8 ? ldx : ld8;
    if (rows * widest >= (1ll << 31)) return fail(BSI_ERR_UNSUPPORTED, "quantize_pack_multi: matrix too large for one launch");
    MultiDst dst = {};
    dst.n_q8 = n_q8_dst;
    dst.n_scales = n_scale_dst;
    for (int i = 0; i < n_q8_dst; ++i) {
        if (q8_dst[i] == nullptr || (reinterpret_cast<uintptr_t>(q8_dst[i]) & 7) != 0)
            return fail(BSI_ERR_INVALID, "quantize_pack_multi: q8 destinations must be non-null and 8-byte aligned");
        dst.q8[i] = q8_dst[i];
    }
    for (int i = 0; i < n_scale_dst; ++i) {
        if (scale_dst[i] == nullptr) return fail(BSI_ERR_INVALID, "quantize_pack_multi: null scale destination");
        dst.scales[i] = scale_dst[i];
    }
    if (int rc = require_sm100()) return rc;
    const double dec_scale = pow(10.0, static_cast<double>(decimal_places));
    uint32_t dec_mult = 0;
    if (decimal_places >= 0 && decimal_places <= 8) {
        dec_mult = 1;
        for (int i = 0; i < decimal_places; ++i) dec_mult *= 10u;
    }
#define BSI_LAUNCH_MULTI(T)                                                                                 \
    do {                                                                                                    \
        const int64_t resident = resident_blocks<quantize_pack_multi_kernel<T>>();                            \
        if (resident <= 0) return BSI_ERR_CUDA;                                                             \
        int64_t blocks = (rows * chunks + 7) / 8;                                                           \
        blocks = blocks < resident ? blocks : resident;                                                     \
        quantize_pack_multi_kernel<T><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(                   \
            static_cast<const T*>(x), static_cast<uint32_t>(rows * chunks), static_cast<uint32_t>(chunks),  \
            static_cast<uint32_t>(ldx), static_cast<uint32_t>(ld8), static_cast<uint32_t>(scale_ld), dec_scale, \
            dec_mult, bits, dst);                                                                    \
    } while (0)
    if (dtype == BSI_DTYPE_F32) BSI_LAUNCH_MULTI(float);
    else if (dtype == BSI_DTYPE_F16) BSI_LAUNCH_MULTI(__half);
    else BSI_LAUNCH_MULTI(__nv_bfloat16);
#undef BSI_LAUNCH_MULTI
    return check_launch("quantize_pack_multi launch");
}

extern "C" int bsi_b200_add_layernorm_pack(const void* x, const void* delta, const void* gamma, const void* beta,
                                           float eps, int dtype, int64_t rows, int64_t H, void* x_out,
                                           int decimal_places, int bits, int n_q8_dst, int8_t* const* q8_dst,
                                           int64_t ld8, int n_scale_dst, float* const* scale_dst, int64_t scale_ld,
                                           bsi_stream_t stream_) {
    using namespace bsi;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (rows < 0 || H <= 0) return fail(BSI_ERR_INVALID, "add_layernorm_pack: bad rows/H");
    if (dtype != BSI_DTYPE_F16 && dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_UNSUPPORTED, "add_layernorm_pack: the layer type must be float16 or bfloat16");
    if ((H & 255) != 0 || H > 16384) return fail(BSI_ERR_UNSUPPORTED, "add_layernorm_pack: H must be a multiple of 256, at most 16384");
    if (bits < 2 || bits > 8) return fail(BSI_ERR_UNSUPPORTED, "add_layernorm_pack: bits must be in [2, 8]");
    if (rows == 0) return BSI_OK;
    if (rows > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "add_layernorm_pack: too many rows");
    if (x == nullptr || gamma == nullptr || beta == nullptr || x_out == nullptr || q8_dst == nullptr || scale_dst == nullptr)
        return fail(BSI_ERR_INVALID, "add_layernorm_pack: null pointer");
    auto misaligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (misaligned(x) || misaligned(x_out) || misaligned(gamma) || misaligned(beta) || (delta != nullptr && misaligned(delta)))
        return fail(BSI_ERR_INVALID, "add_layernorm_pack: pointers must be 16-byte aligned");
    const int64_t chunks = H / 256;
    if (n_q8_dst < 1 || n_q8_dst > BSI_B200_MAX_PEERS || n_scale_dst < 1 || n_scale_dst > BSI_B200_MAX_PEERS ||
        ld8 < H || (ld8 & 7) != 0 || scale_ld < chunks)
        return fail(BSI_ERR_INVALID, "add_layernorm_pack: bad destinations (ld8 >= H, ld8 % 8 == 0, scale_ld >= H/256)");
    MultiDst dst = {};
    dst.n_q8 = n_q8_dst;
    dst.n_scales = n_scale_dst;
    for (int i = 0; i < n_q8_dst; ++i) {
        if (q8_dst[i] == nullptr || (reinterpret_cast<uintptr_t>(q8_dst[i]) & 7) != 0)
            return fail(BSI_ERR_INVALID, "add_layernorm_pack: q8 destinations must be non-null and 8-byte aligned");
        dst.q8[i] = q8_dst[i];
    }
    for (int i = 0; i < n_scale_dst; ++i) {
        if (scale_dst[i] == nullptr) return fail(BSI_ERR_INVALID, "add_layernorm_pack: null scale destination");
        dst.scales[i] = scale_dst[i];
    }
    if (int rc = require_sm100()) return rc;
    const double dec_scale = pow(10.0, static_cast<double>(decimal_places));
    uint32_t dec_mult = 0;
    if (decimal_places >= 0 && decimal_places <= 8) {
        dec_mult = 1;
        for (int i = 0; i < decimal_places; ++i) dec_mult *= 10u;
    }
    const int cpw = static_cast<int>((chunks + 7) / 8);   // chunks per warp, 8 warps
    int64_t blocks = rows;   // one block per row; the kernel's row loop only matters under a block cap
#define BSI_LAUNCH_ALP(T, CPW_)                                                                                   \
    add_layernorm_pack_kernel<T, CPW_><<<static_cast<unsigned>(blocks), 256, 0, stream>>>(                       \
        static_cast<const T*>(x), static_cast<const T*>(delta), static_cast<const T*>(gamma),                    \
        static_cast<const T*>(beta), eps, static_cast<int>(rows), static_cast<int>(H), static_cast<int>(chunks), \
        static_cast<T*>(x_out), dec_scale, dec_mult, bits, ld8, scale_ld, dst)
#define BSI_LAUNCH_ALP_T(T)                       \
    do {                                          \
        if (cpw <= 1) BSI_LAUNCH_ALP(T, 1);       \
        else if (cpw <= 2) BSI_LAUNCH_ALP(T, 2);  \
        else if (cpw <= 4) BSI_LAUNCH_ALP(T, 4);  \
        else BSI_LAUNCH_ALP(T, 8);                \
    } while (0)
    if (dtype == BSI_DTYPE_F16) BSI_LAUNCH_ALP_T(__half);
    else BSI_LAUNCH_ALP_T(__nv_bfloat16);
#undef BSI_LAUNCH_ALP_T
#undef BSI_LAUNCH_ALP
    return check_launch("add_layernorm_pack launch");
}

extern "C" int bsi_b200_decimal_absmax(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx, int decimal_places,
                                       uint64_t* row_absmax, int32_t* row_negative, bsi_stream_t stream_) {
    using namespace bsi;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (rows < 0 || D < 0 || ldx < D) return fail(BSI_ERR_INVALID, "decimal_absmax: bad rows / D / ldx");
    if (rows == 0) return BSI_OK;
    if (x == nullptr || row_absmax == nullptr || row_negative == nullptr) return fail(BSI_ERR_INVALID, "decimal_absmax: null pointer");
    if (dtype != BSI_DTYPE_F32 && dtype != BSI_DTYPE_F16 && dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_INVALID, "decimal_absmax: unknown dtype");
    if (rows > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "decimal_absmax: too many rows for one launch");
    if (int rc = require_sm100()) return rc;
    const double dec_scale = pow(10.0, static_cast<double>(decimal_places));
    const uint32_t dec_mult = (decimal_places >= 0 && decimal_places <= 8) ? static_cast<uint32_t>(dec_scale + 0.5) : 0u;
    const int64_t chunks = (D + 255) / 256;
    const int esz = dtype == BSI_DTYPE_F32 ? 4 : 2;
    const int vec_ok = ((reinterpret_cast<uintptr_t>(x) & 15) == 0 && ((ldx * esz) & 15) == 0) ? 1 : 0;
    const unsigned g = static_cast<unsigned>(rows);
#define BSI_ABSMAX(T) decimal_absmax_kernel<T><<<g, 256, 0, stream>>>(static_cast<const T*>(x), rows, D, ldx, dec_scale, \
                                                                      dec_mult, chunks, vec_ok, reinterpret_cast<u64*>(row_absmax), row_negative)
    if (dtype == BSI_DTYPE_F32) BSI_ABSMAX(float);
    else if (dtype == BSI_DTYPE_F16) BSI_ABSMAX(__half);
    else BSI_ABSMAX(__nv_bfloat16);
#undef BSI_ABSMAX
    return check_launch("decimal_absmax launch");
}

extern "C" int bsi_b200_pack_plain(const void* x, int dtype, int64_t rows, int64_t D, int64_t ldx, int decimal_places,
                                   int slices, uint64_t* words, int8_t* lo8, int8_t* hi8, int64_t ld8, bsi_stream_t stream_) {
    using namespace bsi;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (rows < 0 || D < 0 || ldx < D) return fail(BSI_ERR_INVALID, "pack_plain: bad rows / D / ldx");
    if (slices < 1 || slices > 64) return fail(BSI_ERR_INVALID, "pack_plain: slices must be in [1, 64]");
    if (rows == 0 || D == 0) return BSI_OK;
    if (x == nullptr) return fail(BSI_ERR_INVALID, "pack_plain: null pointer");
    if (dtype != BSI_DTYPE_F32 && dtype != BSI_DTYPE_F16 && dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_INVALID, "pack_plain: unknown dtype");
    const int64_t chunks = (D + 255) / 256;
    if (lo8 == nullptr && hi8 != nullptr) return fail(BSI_ERR_INVALID, "pack_plain: hi8 without lo8");
    if (lo8 != nullptr && (ld8 < chunks * 256 || (ld8 & 15) != 0 || (reinterpret_cast<uintptr_t>(lo8) & 15) != 0 ||
                           (reinterpret_cast<uintptr_t>(hi8) & 15) != 0))
        return fail(BSI_ERR_INVALID, "pack_plain: int8 images need ld8 >= 256*ceil(D/256), ld8 % 16 == 0, 16-byte bases");
    if (int rc = require_sm100()) return rc;
    const double dec_scale = pow(10.0, static_cast<double>(decimal_places));
    const uint32_t dec_mult = (decimal_places >= 0 && decimal_places <= 8) ? static_cast<uint32_t>(dec_scale + 0.5) : 0u;
    const int64_t W = (D + 63) / 64;
    const int esz = dtype == BSI_DTYPE_F32 ? 4 : 2;
    const int vec_ok = ((reinterpret_cast<uintptr_t>(x) & 15) == 0 && ((ldx * esz) & 15) == 0) ? 1 : 0;
    const int64_t blocks = (rows * chunks + 7) / 8;
    if (blocks > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "pack_plain: too many rows for one launch");
    const unsigned g = static_cast<unsigned>(blocks);
#define BSI_PLAIN(T) pack_plain_kernel<T><<<g, 256, 0, stream>>>(static_cast<const T*>(x), rows, D, ldx, dec_scale, dec_mult, \
                                                                  slices, chunks, W, vec_ok, reinterpret_cast<u64*>(words), lo8, hi8, ld8)
    if (dtype == BSI_DTYPE_F32) BSI_PLAIN(float);
    else if (dtype == BSI_DTYPE_F16) BSI_PLAIN(__half);
    else BSI_PLAIN(__nv_bfloat16);
#undef BSI_PLAIN
    return check_launch("pack_plain launch");
}

extern "C" int bsi_b200_recombine_i8(const uint64_t* words, int64_t rows, int bits, int64_t W,
                                     int8_t* q8, int64_t ld8, bsi_stream_t stream_) {
    using namespace bsi;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (rows < 0 || W <= 0) return fail(BSI_ERR_INVALID, "recombine_i8: bad rows/W");
    if (bits < 2 || bits > 8) return fail(BSI_ERR_UNSUPPORTED, "recombine_i8: bits must be in [2, 8]");
    if (rows == 0) return BSI_OK;
    if (words == nullptr || q8 == nullptr) return fail(BSI_ERR_INVALID, "recombine_i8: null pointer");
    const int64_t chunks = (W + 3) / 4;
    if (ld8 < chunks * 256 || (ld8 & 15) != 0 || (reinterpret_cast<uintptr_t>(q8) & 15) != 0)
        return fail(BSI_ERR_INVALID, "recombine_i8: q8 needs ld8 >= 256*ceil(W/4), ld8 % 16 == 0, 16-byte base");
    if (int rc = require_sm100()) return rc;
    const int64_t blocks = (rows * chunks + 7) / 8;
    if (blocks > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "recombine_i8: too many rows for one launch");
    recombine_i8_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        reinterpret_cast<const u64*>(words), rows, bits, W, chunks, q8, ld8);
    return check_launch("recombine_i8 launch");
}

extern "C" int bsi_b200_key_bounds(const int8_t* q8, int64_t ld8, int64_t rows, int64_t chunks, float* bounds,
                                   bsi_stream_t stream_) {
    using namespace bsi;
    if (rows < 0 || chunks <= 0) return fail(BSI_ERR_INVALID, "key_bounds: bad rows / chunks");
    if (rows == 0) return BSI_OK;
    if (q8 == nullptr || bounds == nullptr) return fail(BSI_ERR_INVALID, "key_bounds: null pointer");
    if (ld8 < chunks * 256 || (ld8 & 7) != 0 || (reinterpret_cast<uintptr_t>(q8) & 7) != 0)
        return fail(BSI_ERR_INVALID, "key_bounds: q8 needs 8-byte aligned rows of at least 256 * chunks bytes");
    if (rows > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "key_bounds: too many rows for one launch");
    if (int rc = require_sm100()) return rc;
    key_bounds_kernel<<<static_cast<unsigned>((rows + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream_)>>>(q8, rows, chunks,
                                                                                                       ld8, bounds);
    return check_launch("key_bounds launch");
}

extern "C" int bsi_b200_cast_bias(const float* out, int64_t ldo, const float* bias, int64_t Q, int64_t R,
                                  void* y, int64_t ldy, int y_dtype, bsi_stream_t stream_) {
    using namespace bsi;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (Q < 0 || R < 0 || ldo < R || ldy < R) return fail(BSI_ERR_INVALID, "cast_bias: bad Q/R/ld");
    if (Q == 0 || R == 0) return BSI_OK;
    if (out == nullptr || y == nullptr) return fail(BSI_ERR_INVALID, "cast_bias: null pointer");
    if (int rc = require_sm100()) return rc;
    const int64_t n = Q * ((R + 3) / 4);
    const int64_t blocks = (n + 255) / 256;
    if (blocks > 0x7fffffffll) return fail(BSI_ERR_UNSUPPORTED, "cast_bias: too large for one launch");
    const unsigned g = static_cast<unsigned>(blocks);
    if (y_dtype == BSI_DTYPE_F32)
        cast_bias_kernel<float><<<g, 256, 0, stream>>>(out, ldo, bias, Q, R, static_cast<float*>(y), ldy);
    else if (y_dtype == BSI_DTYPE_F16)
        cast_bias_kernel<__half><<<g, 256, 0, stream>>>(out, ldo, bias, Q, R, static_cast<__half*>(y), ldy);
    else if (y_dtype == BSI_DTYPE_BF16)
        cast_bias_kernel<__nv_bfloat16><<<g, 256, 0, stream>>>(out, ldo, bias, Q, R,
                                                              static_cast<__nv_bfloat16*>(y), ldy);
    else
        return fail(BSI_ERR_INVALID, "cast_bias: unknown y_dtype");
    return check_launch("cast_bias launch");
}
