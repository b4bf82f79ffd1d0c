// Paired-CTA, persistent variant of the int8 tcgen05 dot engine. Included by dot_tcgen05.cu (same
// translation unit: it shares the PTX wrappers and the device status word).
//
// Why pairs: with one CTA per 128 x 256 tile every SM has to pull 48 KB of operands through L2 for
// every 512 cycles of MMA work (96 B/clk/SM), and the L2->SM fabric delivers about half of that.
// Two CTAs of a cluster work on one 256 x BN tile with tcgen05.mma.cta_group::2: each CTA loads its
// own 128 query rows (A) and only HALF of the key rows (B); the pair's tensor cores read B from
// both shared memories. Operand traffic per SM drops to 32 KB per k-block (64 B/clk/SM at full rate).
//
// Why persistent: a pair walks over tiles t = pair, pair + P, ... . Barrier/TMEM set-up happens once,
// the TMA producer runs ahead into the next tile while the epilogue of the current one drains, and
// the result leaves through shared memory as bulk tensor stores that overlap the next tile's MMAs.
//
// Tile = 256 query rows x BN key rows, BN any multiple of 32 up to 256 (float32 output; the 16-bit layer
// epilogues use 64, 128 or 256): tcgen05.mma with M = 256 takes every N that is a multiple of 16.
//
// Roles per CTA (12 warps; register budget moved with setmaxnreg):
//   warps 0, 2    TMA producers, k-blocks in turn (both CTAs; every load signals the LEADER's full barrier)
//   warps 1, 3    MMA issuers, chunks in turn (leader CTA only); warp 1 also TMEM alloc/dealloc (both CTAs)
//   warps 4..11   epilogue: TMEM -> registers, acc = fmaf(float(I), qs[q][c], acc) per chunk in order;
//                 at the end of a tile: finish into smem, bulk tensor stores (scatter, ragged rows: plain stores)
//
// Barriers (same smem offsets in both CTAs):
//   full[s]    leader's copy used: 1 arrival (leader producer, expect_tx of BOTH CTAs' bytes)
//   empty[s]   local in each CTA: tcgen05.commit (multicast to both CTAs) after the stage's MMAs
//   tfull[b]   local in each CTA: multicast commit after a chunk's 8 MMAs
//   tempty[b]  leader's copy used: one arrival per epilogue warp of BOTH CTAs (16)
// The accumulator ring holds 2 or 4 buffers (BN > 128, else): with narrow tiles the MMA issuers run several chunks
// ahead of the epilogue, which takes the barrier round trip off the critical path.
// What bounds a chunk (clock64 marks in every CTA): the MMAs read A and half of B from shared memory at 64 bytes a cycle, 500 + 2 BN
// cycles for the chunk's 8 (600 at 64 columns, 750 at 128, 1000 at 224); with the float32 chain, three instructions per
// accumulator value instead of one, the epilogue is about as long at 256 columns. Beside the chunks a 512 x 8192 x 2048 dot
// spends 1700 cycles on set-up, 1500 until the first k-block has come, 1000 for the chunk behind it, and 5000 on the store phase.
// Split along K (SPLIT = 2 or 4): where the tiles leave most SMs idle, a cluster of SPLIT pairs shares one tile, each
// with a part of the chunks. The chunk terms are integers, so where the bounds of the integer route hold for every warp
// of the tile (the cluster votes before the first MMA) the parts add up in any order to the float32 chain's bits: every
// warp sends its sums through distributed shared memory to the pair that owns the columns, which adds and stores them.
// If a bound fails anywhere, pair 0 does the whole tile on its own with the chain in order, as an unsplit kernel would.
// 512 x 2048 x 8192 (32 tiles of 256 x 128, 2 pairs each): 13.9 us; 64 x 512 x 16384: 10.5.
// All waits are bounded; a timeout raises the abort flag of both CTAs and every role drains out.
#pragma once

namespace pair {

constexpr int kThreads = 384;
constexpr int kEpiWarps = 8;
constexpr int kFirstEpiWarp = 4;
constexpr int kRegsLow = 40;
constexpr int kRegsHigh = 232;
// setmaxnreg.inc draws only on what setmaxnreg.dec returned to the CTA's own pool (threads x registers per thread at
// launch, the latter being 65536 / threads rounded down to a multiple of 8); an increase beyond the pool never returns.
static_assert(kFirstEpiWarp * 32 * kRegsLow + kEpiWarps * 32 * kRegsHigh <= kThreads * ((65536 / kThreads) / 8 * 8),
              "register budget of the warp groups exceeds the CTA's pool");
constexpr long long kWait = 500000000ll;  // ~0.25 s; real waits are microseconds

constexpr int kSmemLimit = 232448;   // 227 KB: the most dynamic shared memory one CTA can opt in to

template <int BN, typename OutT, bool REQ, int SPLIT>
struct Cfg {
    static_assert(BN % 32 == 0 && BN >= 64 && BN <= 256, "tile width: a multiple of 32 in [64, 256]");
    static constexpr int kHalfN = BN / 2;                 // key rows each CTA loads
    static constexpr int kABytes = BM * BK;               // 16 KB
    static constexpr int kBBytes = kHalfN * BK;           // 4 .. 16 KB, a multiple of 1 KB (swizzle atom)
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kStoreBytes = kEpiWarps * 4096;  // one block of 32 rows x 128 bytes per epilogue warp
    static constexpr int kTmemCols = 512;                 // all of TMEM: 1 CTA per SM anyway
    // accumulator ring: buffers start at multiples of the next power of two >= BN (2 or 4 buffers)
    static constexpr int kAccStride = BN > 128 ? 256 : (BN > 64 ? 128 : 64);
    static constexpr int kAccBufs = BN > 128 ? 2 : 4;
    // key scales and bias of the tile's columns
    static constexpr int kColBytes = BN * (4 + static_cast<int>(sizeof(OutT)));
    // chunk-maximum exchange of the re-quantising epilogue: 2 parities x 8 warps x 32 lanes x 2 bytes + 8 counters
    static constexpr int kXchgBytes = REQ ? 2 * kEpiWarps * 32 * 2 + kEpiWarps * 4 : 0;
    static constexpr int kSumBars = SPLIT > 1 ? kEpiWarps : 0;      // arrival of the other parts' sums, per epilogue warp
    static constexpr int kFixedBytes = kStoreBytes + (2 * 9 + 2 * kAccBufs + 2 + kSumBars) * 8 + 16 + kColBytes + kXchgBytes;
    static constexpr int kFit = (kSmemLimit - kFixedBytes) / kStageBytes;
    static constexpr int kStages = kFit > 9 ? 9 : kFit;   // 6 (BN >= 192), 7, 8, 8, 9 (BN = 64)
    static constexpr int kBarriers = 2 * kStages + 2 * kAccBufs + 2 + kSumBars;
    static constexpr int kSmemBytes = kStages * kStageBytes + kStoreBytes + kBarriers * 8 + 16 + kColBytes + kXchgBytes;
    // Two MMA issuers take the chunks in turn. An issuer's wait for a stage could only mistake the previous lap for its
    // own if that lap's chunk were not drained yet, and the accumulator wait in front of it says that chunk
    // cc - kAccBufs is.
    static_assert(kStages / 2 >= kAccBufs, "a ring lap must not be shorter than the accumulator ring");
    static_assert(kStages >= 4 && kSmemBytes <= kSmemLimit, "operand ring does not fit");
    static_assert(2 * kEpiWarps * (SPLIT - 1) * (kHalfN / SPLIT) * 128 <= kStages * kStageBytes, "sums to send and received fit the ring");
    static_assert(kStages * kStageBytes >= kEpiWarps * 4096 * ((kHalfN * static_cast<int>(sizeof(OutT)) + 127) / 128), "the last tile is staged in the ring");
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}

// True in exactly one lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n.reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(pred));
    return pred != 0;
}

// Without release: with it an arrival waits for every memory access the warp has under way, 1000 to 1200 cycles here. Where
// something was written for the other CTAs, a fence of its own stands in front (fence_cluster), in the threads that wrote. Who
// shares these with another kernel orders its own writes likewise (dot_rows_kernel: its receivers wait for the copies).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    // Plain (CTA-scope release) arrive: the ordering that matters here -- TMEM reads done before the
    // accumulator is overwritten -- comes from tcgen05.wait::ld + tcgen05.fence::before_thread_sync.
    // A cluster-scope release would put a full memory barrier into every chunk of the epilogue.
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ void store_flag_cluster(uint32_t cluster_addr, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t leader_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
        : "memory");
}

__device__ __forceinline__ void umma_i8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives on the barrier at this smem offset in BOTH CTAs of the pair once all earlier MMAs are done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint16_t mask) {   // mask: the pair's two CTAs of the cluster
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(bar), "h"(mask)
        : "memory");
}

// M = 256 across the pair.
__host__ __device__ constexpr uint32_t umma_idesc_pair(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(256 >> 4) << 24);
}

struct AbortCtx {
    volatile int* flag;    // this CTA's abort flag
    uint32_t peer_flag;    // cluster address of the peer's
};

__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, const AbortCtx& a, int site) {
    if (mbar_try(bar, parity)) return true;
    long long t0 = 0;
    for (uint32_t spins = 1;; ++spins) {
        if (mbar_try_parked(bar, parity, 20000u)) return true;
        if ((spins & 15u) == 0u) {
            if (*a.flag) return false;
            const long long now = clock64();
            if (t0 == 0) t0 = now;
            if (now - t0 > kWait) {
                *a.flag = 1;
                store_flag_cluster(a.peer_flag, 1);
                fence_cluster();
                atomicCAS(&g_device_status, 0, 16 + site);
                return false;
            }
        }
    }
}

// float(v) for |v| <= 2^22 without a conversion instruction: adding v to the bit pattern of 1.5 * 2^23 gives the
// float 1.5 * 2^23 + v exactly, and subtracting the constant again is exact too. (A chunk accumulator of 8-bit
// operands is at most 256 * 128 * 128 = 2^22 in magnitude.) An integer add and a float add on the full-rate
// pipes instead of one conversion on the slow one.
__device__ __forceinline__ float int_to_float_exact(int32_t v) {
    return __int_as_float(v + 0x4B400000) - 12582912.0f;
}

// ---- finishing 16 bytes of a row: (acc * w) * scale_inv, + bias, ReLU, in the output type ---------------------------
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    return static_cast<uint64_t>(__float_as_uint(lo)) | (static_cast<uint64_t>(__float_as_uint(hi)) << 32);
}
// The values of two adjacent columns; w0, w1: their key scales.
__device__ __forceinline__ float2 scaled2(const float* acc, float w0, float w1, uint64_t scale2) {
    const uint64_t r = mul2(mul2(pack2(acc[0], acc[1]), pack2(w0, w1)), scale2);
    return make_float2(__uint_as_float(static_cast<uint32_t>(r)), __uint_as_float(static_cast<uint32_t>(r >> 32)));
}
// cast, then + cast(bias) with one rounding: a 16-bit add rounds like the float32 add of the two values rounded to 16
// bits (24 >= 2 * 11 + 2), which is what finish<OutT> computes.
__device__ __forceinline__ uint32_t finish2(float2 v, uint32_t b2, bool has_bias, bool relu, __half) {
    __half2 y = __floats2half2_rn(v.x, v.y);
    if (has_bias) y = __hadd2(y, *reinterpret_cast<const __half2*>(&b2));
    uint32_t o = *reinterpret_cast<const uint32_t*>(&y);
    if (relu) o &= ~__hlt2_mask(y, __half2half2(__ushort_as_half(0)));
    return o;
}
__device__ __forceinline__ uint32_t finish2(float2 v, uint32_t b2, bool has_bias, bool relu, __nv_bfloat16) {
    __nv_bfloat162 y = __floats2bfloat162_rn(v.x, v.y);
    if (has_bias) y = __hadd2(y, *reinterpret_cast<const __nv_bfloat162*>(&b2));
    uint32_t o = *reinterpret_cast<const uint32_t*>(&y);
    if (relu) o &= ~__hlt2_mask(y, __bfloat162bfloat162(__ushort_as_bfloat16(0)));
    return o;
}
// colw / colb: the columns' key scales and bias in shared memory, read by every lane at once.
template <typename OutT>
__device__ __forceinline__ uint4 finish16(const float* acc, const float* colw, const OutT* colb, uint64_t scale2, bool has_bias,
                                          bool relu) {
    if constexpr (sizeof(OutT) == 4) {
        const float4 w = *reinterpret_cast<const float4*>(colw);
        float2 a = scaled2(acc, w.x, w.y, scale2), c = scaled2(acc + 2, w.z, w.w, scale2);
        if (has_bias) {
            const float4 b = *reinterpret_cast<const float4*>(colb);
            a.x += b.x; a.y += b.y; c.x += b.z; c.y += b.w;
        }
        return make_uint4(__float_as_uint(relu_if<float>(a.x, relu)), __float_as_uint(relu_if<float>(a.y, relu)),
                          __float_as_uint(relu_if<float>(c.x, relu)), __float_as_uint(relu_if<float>(c.y, relu)));
    } else {
        const float4 w = *reinterpret_cast<const float4*>(colw);
        const float4 v = *reinterpret_cast<const float4*>(colw + 4);
        const uint4 b = *reinterpret_cast<const uint4*>(colb);
        return make_uint4(finish2(scaled2(acc, w.x, w.y, scale2), b.x, has_bias, relu, OutT()),
                          finish2(scaled2(acc + 2, w.z, w.w, scale2), b.y, has_bias, relu, OutT()),
                          finish2(scaled2(acc + 4, v.x, v.y, scale2), b.z, has_bias, relu, OutT()),
                          finish2(scaled2(acc + 6, v.z, v.w, scale2), b.w, has_bias, relu, OutT()));
    }
}
// The same without bias and ReLU, float32.
__device__ __forceinline__ uint4 finish16_plain(const float* acc, const float* colw, uint64_t scale2) {
    const float4 w = *reinterpret_cast<const float4*>(colw);
    const float2 a = scaled2(acc, w.x, w.y, scale2), c = scaled2(acc + 2, w.z, w.w, scale2);
    return make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(c.x), __float_as_uint(c.y));
}
// One value: cast, + cast(bias) (-0.0: none), ReLU (floor -infinity: none). See finish2 for the 16-bit addition.
__device__ __forceinline__ float finish_value(float v, float b, float floor) {
    const float y = __fadd_rn(v, b);
    return y < floor ? 0.0f : y;
}
__device__ __forceinline__ __half finish_value(float v, __half b, float floor) {
    const __half y = __hadd(__float2half_rn(v), b);
    return __half2float(y) < floor ? __ushort_as_half(0) : y;
}
__device__ __forceinline__ __nv_bfloat16 finish_value(float v, __nv_bfloat16 b, float floor) {
    const __nv_bfloat16 y = __hadd(__float2bfloat16_rn(v), b);
    return __bfloat162float(y) < floor ? __ushort_as_bfloat16(0) : y;
}
// 16 bytes of finished values times a factor, rounded to the output type again.
__device__ __forceinline__ uint4 times(uint4 o, float factor, float) {
    return make_uint4(__float_as_uint(__fmul_rn(__uint_as_float(o.x), factor)), __float_as_uint(__fmul_rn(__uint_as_float(o.y), factor)),
                      __float_as_uint(__fmul_rn(__uint_as_float(o.z), factor)), __float_as_uint(__fmul_rn(__uint_as_float(o.w), factor)));
}
__device__ __forceinline__ uint32_t times2(uint32_t v, float factor, __half) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
    const __half2 y = __floats2half2_rn(f.x * factor, f.y * factor);
    return *reinterpret_cast<const uint32_t*>(&y);
}
__device__ __forceinline__ uint32_t times2(uint32_t v, float factor, __nv_bfloat16) {
    const __nv_bfloat162 y = __floats2bfloat162_rn(__uint_as_float(v << 16) * factor, __uint_as_float(v & 0xffff0000u) * factor);
    return *reinterpret_cast<const uint32_t*>(&y);
}
template <typename OutT>
__device__ __forceinline__ uint4 times(uint4 o, float factor, OutT t) {
    return make_uint4(times2(o.x, factor, t), times2(o.y, factor, t), times2(o.z, factor, t), times2(o.w, factor, t));
}
// 16 bytes of finished values plus those of another matrix. A 16-bit add rounds like the float32 add narrowed (see finish2).
__device__ __forceinline__ uint4 plus16(uint4 a, uint4 b, float) {
    auto sum = [](uint32_t p, uint32_t q) { return __float_as_uint(__fadd_rn(__uint_as_float(p), __uint_as_float(q))); };
    return make_uint4(sum(a.x, b.x), sum(a.y, b.y), sum(a.z, b.z), sum(a.w, b.w));
}
__device__ __forceinline__ uint32_t plus2(uint32_t a, uint32_t b, __half) {
    const __half2 y = __hadd2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&y);
}
__device__ __forceinline__ uint32_t plus2(uint32_t a, uint32_t b, __nv_bfloat16) {
    const __nv_bfloat162 y = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&y);
}
template <typename OutT>
__device__ __forceinline__ uint4 plus16(uint4 a, uint4 b, OutT t) {
    return make_uint4(plus2(a.x, b.x, t), plus2(a.y, b.y, t), plus2(a.z, b.z, t), plus2(a.w, b.w, t));
}
__device__ __forceinline__ float cast_bias(float b, float) { return b; }
__device__ __forceinline__ __half cast_bias(float b, __half) { return __float2half_rn(b); }
__device__ __forceinline__ __nv_bfloat16 cast_bias(float b, __nv_bfloat16) { return __float2bfloat16_rn(b); }

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

__device__ __forceinline__ float most4(float4 v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }
__device__ __forceinline__ float most4(float v) { return v; }
__device__ __forceinline__ float sum4(float4 v) { return (v.x + v.y) + (v.z + v.w); }
__device__ __forceinline__ float sum4(float v) { return v; }
template <typename V>
__device__ __forceinline__ V zero_of();
template <>
__device__ __forceinline__ float4 zero_of<float4>() { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
template <>
__device__ __forceinline__ float zero_of<float>() { return 0.0f; }

// Of 32 rows of per-chunk scales (and sums of squares; norms may be null), `units` vectors V each: the largest scale, the
// largest sum of a row's scales, the largest sum of a row's squares, spread over the lanes (the caller takes the maximum over
// them). Eight lanes read neighbouring vectors of a row, with eight rows per lane in flight, so that a load touches 4 rows'
// lines instead of 32 and up to 32 chunks of both arrays take one trip to memory (16 loads in turns of 8: 6400 cycles with
// the reductions, now 3000). The rows' sums are then halved over the lanes, which takes 7 exchanges instead of 24.
template <typename V>
__device__ __forceinline__ void row_stats(const float* qs, int64_t qs_stride, const float* norms, int64_t n_stride,
                                          int first_row, int Q, int units, float& smax, float& ssum, float& u2) {
    const int lane = threadIdx.x & 31;
    const int sub = lane & 7;
    float t[8], n[8];
#pragma unroll
    for (int h = 0; h < 8; ++h) t[h] = n[h] = 0.0f;
    for (int u0 = 0; u0 < units; u0 += 8) {
        V a[8], b[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            const int r = first_row + h * 4 + (lane >> 3);
            const bool in = u0 + sub < units && r < Q;
            a[h] = in ? reinterpret_cast<const V*>(qs + r * qs_stride)[u0 + sub] : zero_of<V>();
            b[h] = in && norms != nullptr ? reinterpret_cast<const V*>(norms + r * n_stride)[u0 + sub] : zero_of<V>();
        }
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            smax = fmaxf(smax, most4(a[h]));
            t[h] += sum4(a[h]);
            n[h] += sum4(b[h]);
        }
    }
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {        // a lane keeps half of its rows, with both lanes' sums
        const bool upper = (lane & d) != 0;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            if (h < d) {
                const float gt = __shfl_xor_sync(0xffffffffu, upper ? t[h] : t[h + d], d), gn = __shfl_xor_sync(0xffffffffu, upper ? n[h] : n[h + d], d);
                t[h] = (upper ? t[h + d] : t[h]) + gt;
                n[h] = (upper ? n[h + d] : n[h]) + gn;
            }
        }
    }
    ssum = t[0];
    u2 = n[0];
}

// The same for one row per lane: kAhead vectors of each array in flight.
template <typename V, int kAhead>
__device__ __forceinline__ void row_of_lane(const float* qs_row, const float* n_row, int units, float& smax,
                                            float& ssum, float& u2) {
    for (int c = 0; c < units; c += kAhead) {
        V a[kAhead], n[kAhead];
#pragma unroll
        for (int h = 0; h < kAhead; ++h) {
            a[h] = c + h < units ? reinterpret_cast<const V*>(qs_row)[c + h] : zero_of<V>();
            n[h] = c + h < units && n_row != nullptr ? reinterpret_cast<const V*>(n_row)[c + h] : zero_of<V>();
        }
#pragma unroll
        for (int h = 0; h < kAhead; ++h) {
            smax = fmaxf(smax, most4(a[h]));
            ssum += sum4(a[h]);
            u2 += sum4(n[h]);
        }
    }
}

// 16-byte-aligned blocks a warp's kCols columns make: of 128-byte rows, the last one of 64-byte rows where that is left
template <typename OutT, int kCols>
__host__ __device__ constexpr int kBlocks() {
    return (kCols * static_cast<int>(sizeof(OutT)) + 127) / 128;
}

// Stores 32 rows (lane = row) x kCols finished columns: out = (acc * w) * scale_inv + bias, ReLU.
// A lane owns a row. Blocks of 32 rows x 128 bytes are finished into shared memory (16-byte pieces swizzled as the
// tensor map wants them, which also keeps the banks apart) and leave as one bulk tensor store each, so that the warp is
// back in the next tile's main loop while they drain; written with ordinary stores, the output took half of a tile's
// time at 16 chunks. A warp has one block of its own; places != nullptr (a CTA's last tile, when nothing reads the operand
// ring any more) gives every block its own place.
// ADD: a matrix is added to the finished values. An instantiation of its own: skipped by a branch, its few instructions still
// cost a 512 x 8192 x 2048 dot 0.5 us, since what runs once per tile waits for its instructions to be fetched.
template <typename OutT, int kCols, bool ADD>
__device__ __forceinline__ void store_columns(const float (&acc)[kCols], uint8_t* places, uint8_t* own, const float* colw, const OutT* colb,
                                              const CUtensorMap& map_o, const CUtensorMap& map_t, OutT* __restrict__ outp, int64_t ldo,
                                              int row_shift, int row_base, int Q, int col, int R, float scale_inv, bool has_bias, bool relu,
                                              const Finishing& fin, int store_flags) {
    const int lane = threadIdx.x & 31;
    constexpr int E = static_cast<int>(sizeof(OutT));
    constexpr int kPerChunk = 16 / E;                        // values per 16-byte piece
    constexpr int kRoundCols = 128 / E;                      // columns per block
    constexpr int kFull = kCols / kRoundCols;                // whole blocks; then one of 64-byte rows, or none
    constexpr int kRounds = kBlocks<OutT, kCols>();
    const uint64_t scale2 = pack2(scale_inv, scale_inv);
    if ((store_flags & 1) && (kCols * E) % 64 == 0) {
        const bool bulk = (store_flags & 4) != 0;
#pragma unroll
        for (int g = 0; g < kRounds; ++g) {
            const bool whole = g < kFull;
            const int nch = whole ? 8 : 4;                   // 16-byte pieces per staged row
            const int cg = g * kRoundCols;
            uint8_t* block = places != nullptr ? places + g * 4096 : own;
            if (bulk && places == nullptr) {
                if (elect_one()) tma_store_wait_read();
                __syncwarp();
            }
            uint8_t* dst = block + lane * (nch * 16);
            // The matrix to add, on its way while the block is finished, neighbouring lanes on neighbouring pieces of a row: loaded
            // behind it, a row per lane, it made the store phase of a 256 x 256 tile twice as long.
            uint4 add[8];
            if constexpr (ADD) {
                const OutT* a = behind_wait(static_cast<const OutT*>(fin.add)) + col + cg + (lane & (nch - 1)) * kPerChunk;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = row_base + i * (32 / nch) + lane / nch;
                    add[i] = make_uint4(0u, 0u, 0u, 0u);
                    if (i < nch && r < Q && col + cg + (lane & (nch - 1)) * kPerChunk < R)
                        add[i] = *reinterpret_cast<const uint4*>(a + static_cast<int64_t>(r) * fin.ld_add);
                }
            }
#pragma unroll
            for (int ch = 0; ch < 8; ++ch) {
                if (ch < nch) {
                    const int swz = whole ? (ch ^ (lane & 7)) : (ch ^ ((lane >> 1) & 3));
                    const int j = cg + ch * kPerChunk;
                    if (j < kCols)
                        *reinterpret_cast<uint4*>(dst + (swz << 4)) = finish16<OutT>(acc + j, colw + j, colb + j, scale2, has_bias, relu);
                }
            }
            if (col + cg < fin.scaled_cols) {      // a second look at the lane's own row, so that other blocks pay one branch
                for (int ch = 0; ch < nch; ++ch) {
                    if (col + cg + ch * kPerChunk >= fin.scaled_cols) break;
                    uint4* o = reinterpret_cast<uint4*>(dst + ((whole ? (ch ^ (lane & 7)) : (ch ^ ((lane >> 1) & 3))) << 4));
                    *o = times(*o, fin.factor, OutT());
                }
            }
            if constexpr (ADD) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < nch) {
                        uint4* o = reinterpret_cast<uint4*>(block + (i * (32 / nch) + lane / nch) * (nch * 16) +
                                                            (((lane & (nch - 1)) ^ (whole ? (i * 4 + (lane >> 3)) & 7 : ((i * 8 + (lane >> 2)) >> 1) & 3)) << 4));
                        *o = plus16(*o, add[i], OutT());     // beyond the matrix: clipped or not stored
                    }
            }
            if (bulk) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (row_base < Q && col + cg < R && elect_one())    // rows and columns beyond the matrix are clipped
                    tma_store_2d(whole ? &map_o : &map_t, smem_u32(block), col + cg, row_base);
            } else {
                __syncwarp();
                const int cchunk = lane & (nch - 1);
                const int c = col + cg + cchunk * kPerChunk;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i < nch) {
                        const int rr = i * (32 / nch) + lane / nch;
                        const int swz = whole ? (cchunk ^ (rr & 7)) : (cchunk ^ ((rr >> 1) & 3));
                        const uint4 o = *reinterpret_cast<const uint4*>(block + rr * (nch * 16) + (swz << 4));
                        const int grow = row_base + rr;
                        if (grow < Q && c < R)               // R is a multiple of kPerChunk on this path
                            *reinterpret_cast<uint4*>(outp + static_cast<int64_t>(grow - row_shift) * ldo + c) = o;
                    }
                }
                __syncwarp();
            }
        }
        return;
    }
    // Rows that do not start on 16 bytes, shares narrower than 64 bytes: blocks of 32 rows x kWide raw sums through the
    // warp's 4 KB, then kWide adjacent columns of 32 / kWide rows at a time, so that a store covers consecutive addresses. A value
    // takes a load, a few multiplications and additions, and a store: no bias is -0.0, which leaves every value as it is, no
    // ReLU a floor of -infinity. With the three questions asked per value it was 40 instructions: 300 x 5001
    // x 1000 11.8 -> 9.1 us, 2973 x 4096 -> 12818 bfloat16 217 -> 165.
    constexpr int kWide = kCols < 32 ? (kCols & -kCols) : 32;
    if (store_flags & 4) {
        if (elect_one()) tma_store_wait_read();
        __syncwarp();
    }
    float* stage = reinterpret_cast<float*>(own);
    const int cj = lane & (kWide - 1);
    const float floor = relu ? 0.0f : -__uint_as_float(0x7f800000u);
#pragma unroll
    for (int g = 0; g < (kCols + kWide - 1) / kWide; ++g) {
#pragma unroll
        for (int j = 0; j < kWide; ++j)
            if (g * kWide + j < kCols) stage[lane * kWide + (j ^ (lane & (kWide - 1)))] = acc[g * kWide + j];
        __syncwarp();
        const int j = g * kWide + cj;
        const bool in = j < kCols && col + j < R;
        const float w = in ? colw[j] : 0.0f;
        const OutT bv = in && has_bias ? colb[j] : cast_bias(-0.0f, OutT());
        const int rows = in ? Q - row_base - lane / kWide : 0;         // this lane's rows are 32 / kWide apart
        const int64_t first = static_cast<int64_t>(row_base - row_shift + lane / kWide) * ldo + col + j;
        OutT* o = outp + first;
        const OutT* a = !ADD ? nullptr : behind_wait(static_cast<const OutT*>(fin.add)) + static_cast<int64_t>(row_base + lane / kWide) * fin.ld_add + col + j;
        const bool scaled = col + g * kWide < fin.scaled_cols;         // any of the group's columns: then each looks for itself
#pragma unroll 1
        for (int i0 = 0; i0 < kWide; i0 += 8) {
            OutT y[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int rr = (i0 + e) * (32 / kWide) + lane / kWide;
                y[e] = finish_value((stage[rr * kWide + (cj ^ (rr & (kWide - 1)))] * w) * scale_inv, bv, floor);
            }
            if (scaled) {
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = scaled_if<OutT>(y[e], col + j < fin.scaled_cols, fin.factor);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if ((i0 + e) * (32 / kWide) < rows) *o = ADD ? plus<OutT>(y[e], *a) : y[e];
                o += (32 / kWide) * ldo;
                if (ADD) a += (32 / kWide) * fin.ld_add;
            }
        }
        __syncwarp();
    }
}

// Folds the last chunk in (accumulators at taddr in tensor memory) and stores the tile, where a pair has one tile (ONE): block
// by block of 32 columns, the next one's accumulators on their way while one is finished, so that the first bulk store leaves 2000
// cycles earlier than with everything folded and turned into floats first. What bounds the rest is shared memory (a block is
// written once and read once) and the stores, 30 bytes a cycle and SM. kind: float32 chain, or int32 sums below 2^22 / 2^24 in
// magnitude. Every block has its own place in the operand ring, which nothing reads any more. done(): called when the
// accumulators have been read. Finished from a rolled loop over raw sums in shared memory, with a third of the code, the same
// dots took 5 to 10 % longer: two more passes over shared memory.
enum SumKind { kFloatSums = 0, kSmallInts = 1, kInts = 2 };
template <typename OutT, int kCols, bool ADD, typename Done>
__device__ __forceinline__ void fold_and_store(const float (&acc)[kCols], uint32_t taddr, float qscale, int kind, uint8_t* places, const float* colw,
                                               const OutT* colb, const CUtensorMap& map_o, const CUtensorMap& map_t, int row_base, int Q,
                                               int col, int R, float scale_inv, bool has_bias, bool relu, const Finishing& fin, Done done) {
    const int lane = threadIdx.x & 31;
    constexpr int E = static_cast<int>(sizeof(OutT));
    constexpr int kPerChunk = 16 / E;
    constexpr int kRoundCols = 128 / E;
    constexpr int kFull = kCols / kRoundCols;
    constexpr int kGroups = (kCols + 31) / 32;               // of 32 columns, the last one of 16 where that is left
    const uint64_t scale2 = pack2(scale_inv, scale_inv);
    const bool plain = E == 4 && !has_bias && !relu;
    const int qmul = kind == kFloatSums ? 0 : __float2int_rn(qscale);
    int32_t v[2][32];
    if (kCols >= 32) tmem_ld32(taddr, v[0]); else tmem_ld16(taddr, v[0]);
    // The matrix to add as in store_columns, from a block's first group to its last (two of 16 bits); four loads of a wide tile's
    // block, for the sake of registers, wait until the block is finished.
    constexpr int kAhead = kCols <= 64 ? 8 : 4;
    uint4 add[kAhead];
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
        const int c0 = g * 32, n = kCols - c0 < 32 ? kCols - c0 : 32;
        int32_t (&now)[32] = v[g & 1];
        tmem_ld_wait_for(now);
        if (g + 1 < kGroups) {
            if (kCols - c0 - 32 >= 32) tmem_ld32(taddr + c0 + 32, v[(g + 1) & 1]); else tmem_ld16(taddr + c0 + 32, v[(g + 1) & 1]);
        } else {
            tc_fence_before();
            done();
        }
        const int round = c0 / kRoundCols, cg = round * kRoundCols;
        const bool whole = round < kFull;
        const int nch = whole ? 8 : 4;
        const int tch = lane & (nch - 1), trow = lane / nch, step = 32 / nch;
        const bool in = col + cg + tch * kPerChunk < R;
        auto fetch = [&](int i) {
            const int r = row_base + trow + i * step;
            if (!in || r >= Q) return make_uint4(0u, 0u, 0u, 0u);
            return *reinterpret_cast<const uint4*>(behind_wait(static_cast<const OutT*>(fin.add)) + static_cast<int64_t>(r) * fin.ld_add + col + cg + tch * kPerChunk);
        };
        if constexpr (ADD) {
            if (c0 == cg) {
#pragma unroll
                for (int i = 0; i < kAhead; ++i)
                    if (i < nch) add[i] = fetch(i);
            }
        }
        float f[32];
        if (kind == kSmallInts) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
                if (e < n) f[e] = int_to_float_exact(now[e] * qmul + __float_as_int(acc[c0 + e]));
        } else if (kind == kInts) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
                if (e < n) f[e] = static_cast<float>(now[e] * qmul + __float_as_int(acc[c0 + e]));
        } else {
#pragma unroll
            for (int e = 0; e < 32; ++e)
                if (e < n) f[e] = __fmaf_rn(int_to_float_exact(now[e]), qscale, acc[c0 + e]);
        }
        uint8_t* block = places + round * 4096;
        uint8_t* dst = block + lane * (whole ? 128 : 64);
        auto finish_pieces = [&](auto with) {
#pragma unroll
            for (int j = 0; j < 32; j += kPerChunk) {
                if (j < n) {
                    const int ch = (c0 + j - cg) / kPerChunk;
                    *reinterpret_cast<uint4*>(dst + ((whole ? (ch ^ (lane & 7)) : (ch ^ ((lane >> 1) & 3))) << 4)) = with(j);
                }
            }
        };
        if (plain) finish_pieces([&](int j) { return finish16_plain(f + j, colw + c0 + j, scale2); });
        else finish_pieces([&](int j) { return finish16<OutT>(f + j, colw + c0 + j, colb + c0 + j, scale2, has_bias, relu); });
        if (c0 + n == cg + kRoundCols || c0 + n == kCols) {
            auto piece = [&](int row, int ch) { return reinterpret_cast<uint4*>(block + row * (nch * 16) + ((whole ? (ch ^ (row & 7)) : (ch ^ ((row >> 1) & 3))) << 4)); };
            if (col + cg < fin.scaled_cols) {      // a second look at the lane's own row, so that other blocks pay one branch
#pragma unroll 1
                for (int ch = 0; ch < nch && col + cg + ch * kPerChunk < fin.scaled_cols; ++ch) *piece(lane, ch) = times(*piece(lane, ch), fin.factor, OutT());
            }
            if constexpr (ADD) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < nch) *piece(trow + i * step, tch) = plus16(*piece(trow + i * step, tch), i < kAhead ? add[i < kAhead ? i : 0] : fetch(i), OutT());
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (row_base < Q && col + cg < R && elect_one())    // rows and columns beyond the matrix are clipped
                tma_store_2d(whole ? &map_o : &map_t, smem_u32(block), col + cg, row_base);
        }
    }
}

// ONE: no more tiles than pairs, bulk stores. An instantiation of its own, because the store phase beside the other one made
// kernels with several tiles per pair 2 to 10 % slower.
template <int BN, bool DBG, typename OutT, bool REQ = false, int SPLIT = 1, bool ADD = false, bool ONE = false>
__global__ void __launch_bounds__(kThreads, 1) dot_i8_tcgen05_pair_kernel(
    const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
    const __grid_constant__ CUtensorMap map_o, const __grid_constant__ CUtensorMap map_t,   // out in boxes of 32 rows x 128 / 64 bytes
    int store_flags,   // bit 0: 16-byte pieces of a row are aligned; bit 1: ReLU; bit 2: map_o and map_t are valid
    const float* __restrict__ qs, int64_t qs_stride, const float* __restrict__ bw0,
    const float* __restrict__ bias, int Q, int R, int chunks, int tiles_m, int tiles_total, float scale_inv,
    void* __restrict__ out, int64_t ldo, int32_t* __restrict__ dbg_iacc, const ScatterDst scatter,
    const RequantDst requant, const Finishing fin, const float* __restrict__ k_abs_sum, float q_abs_max,
    const float* __restrict__ q_sq, int64_t q_sq_stride) {
    static_assert(!ONE || (!DBG && !REQ && SPLIT == 1), "one tile per pair: plain dots and layers");
    using C = Cfg<BN, OutT, REQ, SPLIT>;
    constexpr int kStages = C::kStages;
    constexpr int kCols = BN / 2;              // accumulator columns per epilogue warp: a multiple of 16

    extern __shared__ __align__(1024) uint8_t smem[];     // swizzled operand tiles start on 1 KB
    uint8_t* store_area = smem + kStages * C::kStageBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(store_area + C::kStoreBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kBarriers);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* colw = reinterpret_cast<float*>(tmem_slot + 4);                                  // [BN]
    OutT* colb = reinterpret_cast<OutT*>(colw + BN);                                        // [BN]
    uint16_t* xchg_vals = reinterpret_cast<uint16_t*>(colb + BN);                           // [2][kEpiWarps][32] (REQ)
    volatile uint32_t* xchg_count = reinterpret_cast<volatile uint32_t*>(xchg_vals + 2 * kEpiWarps * 32);   // [kEpiWarps]

    // let the next kernel of the stream start its own set-up as soon as every CTA of this grid is running
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
    constexpr int kAccBufs = C::kAccBufs;
    auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * kStages + b); };
    auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * kStages + kAccBufs + b); };

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t drain_bar = bar_base + 8u * (2 * kStages + 2 * kAccBufs + ((warp >> 1) & 1));   // one per issuer
    const uint32_t crank = cluster_ctarank();
    const uint32_t rank = crank & 1u;                     // within the pair
    const uint32_t lead = crank & ~1u;                    // the pair's leader CTA
    const int part = static_cast<int>(crank >> 1);        // of the chunks (SPLIT > 1)
    const uint16_t pair_mask = static_cast<uint16_t>(3u << lead);
    const bool leader = rank == 0;
    const int pair_id = static_cast<int>(blockIdx.x) / (2 * SPLIT);
    const int num_pairs = static_cast<int>(gridDim.x) / (2 * SPLIT);     // split: one tile per cluster
    const int per_part = (chunks + SPLIT - 1) / SPLIT;
    const int c_lo = SPLIT > 1 ? min(part * per_part, chunks) : 0;
    const int my_chunks = SPLIT > 1 ? min(c_lo + per_part, chunks) - c_lo : chunks;
    int num_kb = my_chunks * 2;
    volatile int* vote = reinterpret_cast<volatile int*>(tmem_slot + 2);   // some warp of the cluster has no bound
    const bool has_bias = bias != nullptr;
    const bool relu = (store_flags & 2) != 0;

    const uint32_t leader_full0 = map_to_cta(full_bar(0), lead);
    AbortCtx actx;
    actx.flag = abort_flag;
    actx.peer_flag = map_to_cta(smem_u32(const_cast<int*>(abort_flag)), crank ^ 1u);

    if (warp == 0) {
        // one barrier per lane: full[s], empty[s], tfull[b] and drain count 1 arrival, tempty[b] one per epilogue
        // warp of both CTAs
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
            *abort_flag = 0;
            *vote = 0;
        }
        if (REQ && lane < kEpiWarps) xchg_count[lane] = 0u;
        for (int i = lane; i < C::kBarriers; i += 32) {
            const bool is_tempty = i >= 2 * kStages + kAccBufs && i < 2 * kStages + 2 * kAccBufs;
            mbar_init(bar_base + 8u * i, is_tempty ? 2 * kEpiWarps : 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    // Cluster barrier split around the TMEM allocation: arrive now (warp 0's barrier inits are
    // released by its own arrive, the others have written nothing), wait after the allocation, so the two latencies overlap.
    if (warp == 0) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    else cluster_arrive();
    const bool is_producer = warp == 0 || warp == 2;
    uint32_t tmem_base = 0;
    if (is_producer) {
        // The producers need the barriers of both CTAs, not the accumulator memory: they go on to their
        // first copies while warp 1 is still allocating TMEM.
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        if (warp == 1) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                         ::"r"(smem_u32(tmem_slot)), "r"(static_cast<uint32_t>(C::kTmemCols)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
        tc_fence_before();
        // the issuers and the eight epilogue warps: the TMEM address is in shared memory from here on
        asm volatile("bar.sync 1, %0;" ::"n"((2 + kEpiWarps) * 32) : "memory");
        // both CTAs' barriers are initialised before anyone touches the peer's
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        tc_fence_after();
        tmem_base = *tmem_slot;
    }

    // Programmatic dependent launch: everything above (barriers, TMEM, tensor-map prefetch) touched no global
    // memory of an earlier kernel and may run while that kernel drains; from here on its results are needed.
    // Without the launch attribute both instructions do nothing.
    asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp < kFirstEpiWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsLow));
        if (is_producer) {
            // ---------------- TMA producers ----------------
            // Warps 0 and 2 take the k-blocks in turn. The whole warp walks the loop, as the issuers do, with stage, parity and
            // coordinates carried along, and one elected lane issues.
            constexpr int kProducers = 2;
            const int me = warp >> 1;
            int s = me, kb = me;                       // stage of this warp's next k-block, the k-block
            uint32_t ph = 1;
            bool ok = true;
            auto load = [&](int x, int ya, int yb) {
                ok = __all_sync(0xffffffffu, wait_or_abort(empty_bar(s), ph, actx, 1));
                if (!ok) return;
                if (elect_one()) {
                    const uint32_t a_dst = smem_base + s * C::kStageBytes, bar = leader_full0 + 8u * s;
                    if (leader) mbar_expect_tx(full_bar(s), 2u * C::kStageBytes);
                    tma_load_2d_pair(a_dst, &map_a, x, ya, bar);
                    tma_load_2d_pair(a_dst + C::kABytes, &map_b, x, yb, bar);
                }
                __syncwarp();
                s += kProducers;
                if (s >= kStages) { s -= kStages; ph ^= 1u; }
            };
            for (int tile = pair_id; tile < tiles_total && ok; tile += num_pairs) {
                const int ya = tile % tiles_m * 256 + static_cast<int>(rank) * BM;
                const int yb = tile / tiles_m * BN + static_cast<int>(rank) * C::kHalfN;
                if constexpr (SPLIT > 1) {
                    // the first ring round goes out before the vote: it is the part's own beginning either way
                    const int done = min(kStages, num_kb);
                    cluster_arrive();
                    for (; kb < done && ok; kb += kProducers) load((c_lo * 2 + kb) * BK, ya, yb);
                    cluster_wait();
                    if (*vote) num_kb = part == 0 ? 2 * chunks : done;
                } else {
                    kb = me;
                }
                for (; kb < num_kb && ok; kb += kProducers) load((c_lo * 2 + kb) * BK, ya, yb);
            }
        } else {
            // The vote is the epilogue's; the chunks that the accumulators hold go before it, the part's own beginning either way.
            if constexpr (SPLIT > 1) cluster_arrive();
            const int mi = warp >> 1;
            int total = my_chunks;
            const int early = SPLIT > 1 ? min(kAccBufs, my_chunks) : 0;
            auto voted = [&] {
                cluster_wait();
                if (*vote) total = part == 0 ? chunks : 0;
            };
            if (leader) {
            // ---------------- MMA issuers (leader CTA) ----------------
            // The whole warp walks the loop (so that addresses and descriptors stay in the uniform
            // datapath) and one elected lane issues the tensor-core instructions. A chunk takes an issuer about 500
            // cycles (three barrier waits, eight MMAs, three commits), the MMAs 500 + 2 per column of the tile (A and half of B
            // from shared memory at 64 bytes a cycle), so warps 1 and 3 issue alternate chunks; they share nothing but the
            // order of the rings.
            constexpr uint32_t idesc = umma_idesc_pair(BN);
            if constexpr (SPLIT == 1) total = ((tiles_total - pair_id + num_pairs - 1) / num_pairs) * my_chunks;
            int s = 2 * mi;
            uint32_t ph = 0;
            bool ok = true;
            int cc = mi;
            auto issue = [&](int upto) {
            for (; cc < upto && ok; cc += 2) {
                const int b = cc % kAccBufs;
                const uint32_t tph = static_cast<uint32_t>(cc / kAccBufs) & 1u;
                if (!wait_or_abort(tempty_bar(b), tph ^ 1u, actx, 3)) { ok = false; break; }
                const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(b * C::kAccStride);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    if (!wait_or_abort(full_bar(s), ph, actx, 2)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_base + s * C::kStageBytes;
                    const uint64_t adesc = umma_desc(a_addr);
                    const uint64_t bdesc = umma_desc(a_addr + C::kABytes);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) {
                            umma_i8_pair(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc,
                                         (half | k) != 0 ? 1u : 0u);
                        }
                        umma_commit_pair(empty_bar(s), pair_mask);
                        if (half == 1) umma_commit_pair(tfull_bar(b), pair_mask);
                    }
                    __syncwarp();
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
                s += 2;                                    // the other issuer's chunk
                if (s >= kStages) { s -= kStages; ph ^= 1u; }
            }
            };
            if constexpr (SPLIT > 1) {
                issue(early);
                voted();
            }
            issue(total);
            if (SPLIT > 1 && total == 0 && mi == 0)        // copies that no MMA waited for have to land before the CTAs go
                for (int st = 2 * early; st < min(kStages, num_kb); ++st)
                    if (!wait_or_abort(full_bar(st), 0, actx, 2)) break;
            if (!ok && lane == 0) {
                umma_commit(drain_bar);
                const long long t0 = clock64();
                while (!mbar_try(drain_bar, 0) && clock64() - t0 < kWait / 64) {}
            }
            } else if constexpr (SPLIT > 1) {
                voted();
            }
            if (SPLIT > 1 && total == 0)                   // likewise the MMAs whose sums nobody reads
                for (int cc = mi; cc < early; cc += 2)
                    if (!wait_or_abort(tfull_bar(cc), 0, actx, 4)) break;
            __syncwarp();
        }
        if constexpr (SPLIT > 1) cluster_sync_all();      // the operand rings are free
        __syncwarp();
        cluster_arrive();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsHigh));
        // ---------------- epilogue ----------------
        const int ew = warp - kFirstEpiWarp;   // 0..7
        const int quad = warp & 3;             // TMEM lane quadrant this warp may read
        const int half = ew >> 2;              // which half of the BN columns
        const int col0 = half * kCols;
        uint8_t* my_store = store_area + ew * 4096;
        const uint32_t leader_tempty0 = map_to_cta(tempty_bar(0), lead);

        float acc[kCols];
        int cc = 0;
        bool ok = true;
        uint32_t tiles_done = 0;   // tiles this warp has re-quantised (the chunk-maximum exchange counts them)
        // An aborting warp stays in the loop for its barriers: the four warps of a column half meet at two per tile.
        for (int tile = pair_id; tile < tiles_total; tile += num_pairs) {
            const int tm = tile % tiles_m;
            const int tn = tile / tiles_m;
            const int row = tm * 256 + static_cast<int>(rank) * BM + quad * 32 + lane;
            const int n0 = tn * BN;
            const bool row_ok = row < Q;
            const float* qs_row = behind_wait(qs) + static_cast<int64_t>(row_ok ? row : 0) * (qs_stride ? qs_stride : 1);
#pragma unroll
            for (int j = 0; j < kCols; ++j) acc[j] = 0.0f;
            // Key scale and bias of the column this lane puts into shared memory for the store phase: a quarter of the
            // half's columns per warp, loaded here so that the latency hides behind the main loop.
            constexpr int kOwn = kCols / 4;
            const int own = quad * kOwn + lane;
            float own_w = 0.0f, own_b = 0.0f;
            if (lane < kOwn && n0 + col0 + own < R) {
                own_w = behind_wait(bw0)[n0 + col0 + own];
                if (has_bias) own_b = behind_wait(bias)[n0 + col0 + own];
            }

            // The chunk scale of the next chunk is loaded a whole chunk ahead, the first one in front of the bounds: a scattered load per
            // lane (32 rows) that would otherwise stand in front of every fold.
            float qnext = qs_row[qs_stride ? min(c_lo, chunks - 1) : 0];

            // Integer accumulation where it provably equals the float32 chain: the chunk terms I_c * 2^shift are
            // integers, so while every prefix sum stays below 2^24 in magnitude no float32 addition rounds and
            // acc += I_c << shift in int32 gives the same bits. With A the largest query magnitude, a prefix is at
            // most A x (largest 2^shift of the row) x (sum of |k| over the key row), and also at most
            // A x (sum of the row's 2^shift) x (largest sum of |k| over one chunk of the key row); the key sums come
            // from the caller (k_abs_sum: R row sums, then R chunk maxima, then R sums of squares; null: not
            // available). Where both fail and the query image carries its chunk sums of squares (q_sq), the
            // Cauchy-Schwarz product of the two rows' L2 norms is tried. The test is made for the warp's 32 rows x
            // kCols columns at once, so the branch is uniform; a warp whose bounds all fail runs the float32 chain.
            // Everything the bounds read is loaded in one go: one after the other, as scalars behind the previous
            // bound's outcome, they cost 5 to 10 thousand cycles per tile.
            bool exact = false, small = false;
            if (k_abs_sum != nullptr && ok) {
                // of the warp's key rows: the largest sum of |k| over a row and over one chunk, the largest sum of k^2
                const float* k_sums = behind_wait(k_abs_sum);
                constexpr int kPer = (kCols + 31) / 32;       // key rows per lane
                float kv[3][kPer];
#pragma unroll
                for (int e = 0; e < kPer; ++e) {
                    const int col = min(n0 + col0 + min(e * 32 + lane, kCols - 1), R - 1);
                    kv[0][e] = k_sums[col];
                    kv[1][e] = k_sums[R + col];
                    kv[2][e] = k_sums[2 * static_cast<int64_t>(R) + col];
                }
                // of the warp's query rows: the largest and the largest summed 2^shift of a row, the largest sum of squares
                float smax = 0.0f, ssum = 0.0f, u2 = 0.0f;
                const int first_row = row - lane;
                const float* norms = qs_stride && q_sq != nullptr ? behind_wait(q_sq) : nullptr;
                if (!qs_stride) {
                    if (row_ok) smax = *qs_row;
                    ssum = smax * static_cast<float>(chunks);
                } else {
                    const bool vec = (chunks & 3) == 0 && (qs_stride & 3) == 0 && (q_sq_stride & 3) == 0 &&
                                     ((reinterpret_cast<uintptr_t>(qs) | reinterpret_cast<uintptr_t>(norms)) & 15) == 0;
                    if (chunks > 16) {
                        if (vec) row_stats<float4>(behind_wait(qs), qs_stride, norms, q_sq_stride, first_row, Q, chunks / 4, smax, ssum, u2);
                        else row_stats<float>(behind_wait(qs), qs_stride, norms, q_sq_stride, first_row, Q, chunks, smax, ssum, u2);
                    } else if (row_ok) {
                        // few chunks: a row per lane, everything in one go or two
                        const float* nrow = norms != nullptr ? norms + static_cast<int64_t>(row) * q_sq_stride : nullptr;
                        if (vec) row_of_lane<float4, 4>(qs_row, nrow, chunks / 4, smax, ssum, u2);
                        else row_of_lane<float, 8>(qs_row, nrow, chunks, smax, ssum, u2);
                    }
                }
                float ktot = kv[0][0], kchk = kv[1][0], k2 = kv[2][0];
#pragma unroll
                for (int e = 1; e < kPer; ++e) {
                    ktot = fmaxf(ktot, kv[0][e]);
                    kchk = fmaxf(kchk, kv[1][e]);
                    k2 = fmaxf(k2, kv[2][e]);
                }
                // An infinity anywhere fails the test. By shuffles, all six maxima side by side: with redux.sync (nvcc 12.9) an earlier form of this code
                // had norm = 0 in every warp of one instantiation (256 columns, four parts), and so exact sums beyond 2^24.
                // Not a divergent warp (a __syncwarp before each changed nothing) nor wrong operands (the other four maxima
                // were right, and shuffles of the same registers are); writing the operands out made it go away. The split
                // test has a row beyond the bounds for every width and number of parts.
                float most[6] = {smax, ssum, u2, ktot, kchk, k2};
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) {
                    float got[6];
#pragma unroll
                    for (int e = 0; e < 6; ++e) got[e] = __shfl_xor_sync(0xffffffffu, most[e], d);
#pragma unroll
                    for (int e = 0; e < 6; ++e) most[e] = fmaxf(most[e], got[e]);
                }
                // the sums above round (relative 2^-24 per addition, at most a few thousand additions): 0.999 covers it
                const float first = fminf(most[0] * most[3], most[1] * most[4]) * q_abs_max;
                const float norm = q_sq != nullptr && qs_stride ? most[2] * most[5] : __uint_as_float(0x7f800000u);
                exact = first < 16777216.0f * 0.999f || norm < 281474976710656.0f * 0.999f;      // 2^24, 2^48
                small = first < 4194304.0f * 0.999f || norm < 17592186044416.0f * 0.999f;        // 2^22, 2^44
            }

            int n_chunks = my_chunks;
            bool whole_tile = SPLIT == 1;      // this pair does all chunks and stores all columns
            if constexpr (SPLIT > 1) {
                if (!exact && lane < 2 * SPLIT) {
                    store_flag_cluster(map_to_cta(smem_u32(const_cast<int*>(vote)), static_cast<uint32_t>(lane)), 1);
                    fence_cluster();
                }
                __syncwarp();
                cluster_sync_all();
                if (*vote) {
                    whole_tile = part == 0;
                    n_chunks = part == 0 ? chunks : 0;
                }
            }
            // The last round of accumulators has no user after this one, and its arrivals could reach the leader after its end.
            const int hand_back = (SPLIT > 1 ? n_chunks : (tiles_total - pair_id + num_pairs - 1) / num_pairs * my_chunks) - kAccBufs;
            const int here = ONE ? n_chunks - 1 : n_chunks;      // the store phase has the last one
            for (int c = 0; c < here && ok; ++c, ++cc) {
                const int b = cc % kAccBufs;
                const uint32_t tph = static_cast<uint32_t>(cc / kAccBufs) & 1u;
                const float qscale = qnext;
                if (qs_stride && c + 1 < n_chunks) qnext = qs_row[c_lo + c + 1];
                const int qmul = exact ? __float2int_rn(qscale) : 0;
                if (!wait_or_abort(tfull_bar(b), tph, actx, 4)) { ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                                       static_cast<uint32_t>(b * C::kAccStride + col0);
                // The warp's kCols columns come in pieces of up to 64 (two loads issued back to back, one wait):
                // under the tensor pipe's own accumulator traffic a TMEM load takes a few hundred cycles, and the
                // fewer round trips a chunk needs, the sooner its buffer goes back to the MMA issuer. While this
                // warp waits, the other epilogue warp of the SM sub-partition folds its piece.
                int32_t v[2][32];
                constexpr int kSuper = (kCols + 63) / 64;
#pragma unroll
                for (int sp = 0; sp < kSuper; ++sp) {
                    const int c0 = sp * 64;
                    const int wsp = (kCols - c0) < 64 ? (kCols - c0) : 64;   // 64, 48, 32 or 16
                    if (wsp >= 32) tmem_ld32(taddr + c0, v[0]); else tmem_ld16(taddr + c0, v[0]);
                    if (wsp == 64) tmem_ld32(taddr + c0 + 32, v[1]);
                    else if (wsp == 48) tmem_ld16(taddr + c0 + 32, v[1]);
                    tmem_ld_wait();
                    if (sp + 1 == kSuper) {
                        // every column of the buffer is in registers: hand it back before the last piece is folded in
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0 && cc < hand_back) mbar_arrive_cluster(leader_tempty0 + 8u * b);
                    }
                    if (exact) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                if (h * 32 + e < wsp)
                                    acc[c0 + h * 32 + e] =
                                        __int_as_float(v[h][e] * qmul + __float_as_int(acc[c0 + h * 32 + e]));
                            }
                        }
                    } else {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                if (h * 32 + e < wsp)
                                    acc[c0 + h * 32 + e] = __fmaf_rn(int_to_float_exact(v[h][e]), qscale, acc[c0 + h * 32 + e]);
                            }
                        }
                    }
                    if (DBG) {
                        if (row_ok) {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
#pragma unroll
                                for (int e = 0; e < 32; ++e) {
                                    const int col = n0 + col0 + c0 + h * 32 + e;
                                    if (h * 32 + e < wsp && col < R)
                                        dbg_iacc[(static_cast<int64_t>(row) * R + col) * chunks + c] = v[h][e];
                                }
                            }
                        }
                    }
                }
            }
            if constexpr (!REQ && SPLIT == 1 && !ONE) {
                __syncwarp();
                if (tile + num_pairs >= tiles_total) cluster_arrive();
            }
            // the half's key scales and bias into shared memory: behind the first barrier nobody reads the last tile's
            asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
            if (lane < kOwn) {
                colw[col0 + own] = own_w;
                colb[col0 + own] = cast_bias(own_b, OutT());
            }
            asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
            if constexpr (SPLIT > 1) {
                constexpr int kShare = kCols / SPLIT;        // columns of this warp that each pair stores
                const bool add_up = *vote == 0;
                __syncwarp();
                cluster_sync_all();          // the operand rings of all CTAs are free
                // Sums to send and sums received, both [warp][slot][4 columns][lane] in the ring: 512 bytes per 4 columns,
                // no bank conflicts. A share travels as one bulk copy; stored to the other CTA's shared memory by the
                // lanes, the exchange of a 256-column tile took 8 us.
                constexpr int kShareBytes = kShare * 128, kSlotBytes = (SPLIT - 1) * kShareBytes;
                const uint32_t sum_bar = bar_base + 8u * (2 * kStages + 2 * kAccBufs + 2 + ew);
                uint8_t* to_send = smem + ew * kSlotBytes;
                uint8_t* received = smem + (kEpiWarps + ew) * kSlotBytes;
                if (add_up && ok) {
                    if (lane == 0) mbar_expect_tx(sum_bar, kSlotBytes);
#pragma unroll
                    for (int q = 0; q < SPLIT; ++q) {
                        if (q != part) {
                            uint8_t* mine = to_send + (q < part ? q : q - 1) * kShareBytes + lane * 16;
#pragma unroll
                            for (int j = 0; j < kShare; j += 4)
                                *reinterpret_cast<float4*>(mine + j * 128) = make_float4(acc[q * kShare + j], acc[q * kShare + j + 1],
                                                                                         acc[q * kShare + j + 2], acc[q * kShare + j + 3]);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane < SPLIT && lane != part) {
                        const uint32_t cta = static_cast<uint32_t>(2 * lane) + rank;
                        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                     ::"r"(map_to_cta(smem_u32(received), cta) + static_cast<uint32_t>((part < lane ? part : part - 1) * kShareBytes)),
                                     "r"(smem_u32(to_send) + static_cast<uint32_t>((lane < part ? lane : lane - 1) * kShareBytes)), "r"(kShareBytes),
                                     "r"(map_to_cta(sum_bar, cta)) : "memory");
                    }
                    __syncwarp();
                    ok = wait_or_abort(sum_bar, 0, actx, 6);
                }
                __syncwarp();
                cluster_arrive();
                if (add_up) {
                    if (!ok) continue;
                    int sum[kShare];
#pragma unroll
                    for (int q = 0; q < SPLIT; ++q) {
                        if (q == part) {
#pragma unroll
                            for (int j = 0; j < kShare; ++j) sum[j] = __float_as_int(acc[q * kShare + j]);
                        }
                    }
#pragma unroll
                    for (int q = 0; q < SPLIT - 1; ++q) {
#pragma unroll
                        for (int j = 0; j < kShare; j += 4) {
                            const int4 v = *reinterpret_cast<const int4*>(received + lane * 16 + (q * kShare + j) * 128);
                            sum[j] += v.x; sum[j + 1] += v.y; sum[j + 2] += v.z; sum[j + 3] += v.w;
                        }
                    }
                    if (lane == 0) atomicAdd(&g_exact_int_tiles, 1ull);
                    float val[kShare];
#pragma unroll
                    for (int j = 0; j < kShare; ++j) val[j] = small ? int_to_float_exact(sum[j]) : static_cast<float>(sum[j]);
                    const int cs = col0 + part * kShare;
                    store_columns<OutT, kShare, ADD>(val, nullptr, my_store, colw + cs, colb + cs, map_o, map_t, static_cast<OutT*>(out), ldo, 0,
                                                tm * 256 + static_cast<int>(rank) * BM + quad * 32, Q, n0 + cs, R, scale_inv, has_bias, relu,
                                                fin, store_flags);
                    continue;
                }
                if (!whole_tile) continue;
            }
            const int row_base = tm * 256 + static_cast<int>(rank) * BM + quad * 32;
            if constexpr (ONE) {
                const int b = cc % kAccBufs;
                ok = __all_sync(0xffffffffu, ok && wait_or_abort(tfull_bar(b), static_cast<uint32_t>(cc / kAccBufs) & 1u, actx, 4));
                if (!ok) {
                    cluster_arrive();
                    break;
                }
                tc_fence_after();
                if (exact && lane == 0) atomicAdd(&g_exact_int_tiles, 1ull);
                fold_and_store<OutT, kCols, ADD>(acc, tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(b * C::kAccStride + col0),
                                                 qnext, !exact ? kFloatSums : small ? kSmallInts : kInts, smem + ew * kBlocks<OutT, kCols>() * 4096,
                                                 colw + col0, colb + col0, map_o, map_t, row_base, Q, n0 + col0, R, scale_inv, has_bias, relu, fin,
                                                 [] { __syncwarp(); cluster_arrive(); });
                break;
            }
            if (!ok) continue;
            if (exact) {
                // the int32 sums (below 2^24 in magnitude) as floats: what the float32 chain would hold. Below 2^22 by an
                // integer and a float add, at four times the rate of the conversion instruction.
                if (small) {
#pragma unroll
                    for (int j = 0; j < kCols; ++j) acc[j] = int_to_float_exact(__float_as_int(acc[j]));
                } else {
#pragma unroll
                    for (int j = 0; j < kCols; ++j) acc[j] = static_cast<float>(__float_as_int(acc[j]));
                }
                if (lane == 0) atomicAdd(&g_exact_int_tiles, 1ull);
            }

            // ---- tile result: out = (acc * bw0[r]) * scale_inv ----
            if constexpr (REQ) {
                static_assert(BN == 256 && !DBG && sizeof(OutT) == 2, "re-quantisation: 256-wide tiles, 16-bit layer type");
                {
                    // ---- fused re-quantisation: the finished value in the layer's type (cast + bias, ReLU) is
                    // what the next linear's packer would read; with BN = 256 a tile row is exactly one chunk,
                    // split between this warp and the warp of the other column half. Same integers as the pack
                    // kernel's fast path (the values have 16-bit precision, so the float32 rounding is exact).
                    const uint64_t scale2 = pack2(scale_inv, scale_inv);
                    RawLane<OutT> y[kCols / 8];
                    uint32_t amax_bits = 0;                   // pattern of OutT: orders like the magnitude
#pragma unroll
                    for (int j = 0; j < kCols / 8; ++j) {
                        y[j].v[0] = finish16<OutT>(acc + j * 8, colw + col0 + j * 8, colb + col0 + j * 8, scale2, has_bias, relu);
                        amax_bits = max(amax_bits, y[j].abs_max());
                    }
                    // Largest magnitude of the whole chunk: swap with the partner warp (same rows, other column
                    // half). The value is one of the OutT values, so its 16-bit pattern carries it exactly. Each
                    // warp publishes into its slot of parity (tiles_done & 1) and bumps its counter; a slot is
                    // rewritten two tiles later, after the partner's next publication, which follows its read.
                    // The wait is bounded like every other wait of the kernel.
                    {
                        const uint32_t par = tiles_done & 1u;
                        xchg_vals[(par * kEpiWarps + ew) * 32 + lane] = static_cast<uint16_t>(amax_bits);
                        __syncwarp();
                        if (lane == 0) {
                            __threadfence_block();
                            xchg_count[ew] = tiles_done + 1u;
                        }
                        const long long t0 = clock64();
                        while (static_cast<int32_t>(xchg_count[ew ^ 4] - (tiles_done + 1u)) < 0) {
                            if (*actx.flag || clock64() - t0 > kWait) {
                                *actx.flag = 1;
                                store_flag_cluster(actx.peer_flag, 1);
                                fence_cluster();
                                atomicCAS(&g_device_status, 0, 16 + 7);
                                ok = false;
                                break;
                            }
                        }
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) continue;
                        __threadfence_block();
                        amax_bits = max(amax_bits, static_cast<uint32_t>(xchg_vals[(par * kEpiWarps + (ew ^ 4)) * 32 + lane]));
                        ++tiles_done;
                    }
                    float amax = RawLane<OutT>::abs_value(amax_bits);
                    if (!(amax * requant.mult < 8388608.0f)) {      // NaN fails the comparison too
                        // NaN / inf / out of the exact range: not representable on this path; report, store zeros
                        atomicCAS(&g_device_status, 0, 48);
                        amax = 0.0f;
#pragma unroll
                        for (int j = 0; j < kCols / 8; ++j) y[j].v[0] = make_uint4(0u, 0u, 0u, 0u);
                    }
                    const int shift = fast_shift(amax, requant.mult, requant.bits);
                    // stage 32 rows x 128 bytes through this warp's 4 KB (16-byte chunks XOR-swizzled by row)
                    uint8_t* dst = my_store + lane * 128;
#pragma unroll
                    for (int ch = 0; ch < 8; ++ch) {
                        const u64 lo = y[2 * ch].quantise(requant.mult, shift, requant.bits);
                        const u64 hi = y[2 * ch + 1].quantise(requant.mult, shift, requant.bits);
                        *reinterpret_cast<uint4*>(dst + ((ch ^ (lane & 7)) << 4)) =
                            make_uint4(static_cast<uint32_t>(lo), static_cast<uint32_t>(lo >> 32), static_cast<uint32_t>(hi),
                                       static_cast<uint32_t>(hi >> 32));
                    }
                    __syncwarp();
                    const int cchunk = lane & 7;
                    const int col = n0 + col0 + cchunk * 16;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int rr = i * 4 + (lane >> 3);
                        const uint4 o = *reinterpret_cast<const uint4*>(my_store + rr * 128 + ((cchunk ^ (rr & 7)) << 4));
                        const int grow = row_base + rr;
                        if (grow < Q) {
                            const int64_t off = static_cast<int64_t>(grow) * requant.ld8 + col;
#pragma unroll
                            for (int d = 0; d < BSI_B200_MAX_PEERS; ++d)
                                if (d < requant.n) *reinterpret_cast<uint4*>(requant.q8[d] + off) = o;
                        }
                    }
                    if (half == 0 && row_ok) {
                        const float scale = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);   // 2^shift
                        const int64_t off = static_cast<int64_t>(row) * requant.scale_ld + (n0 >> 8);
#pragma unroll
                        for (int d = 0; d < BSI_B200_MAX_PEERS; ++d)
                            if (d < requant.n) requant.scales[d][off] = scale;
                    }
                    __syncwarp();
                    continue;
                }
            }
            OutT* outp = static_cast<OutT*>(out);
            int row_shift = 0;   // first global row of the destination matrix this warp's 32 rows belong to
            if (scatter.n > 0) {
                int d = row_base / scatter.rows_per_dst;
                d = d < scatter.n ? d : scatter.n - 1;
                outp = static_cast<OutT*>(scatter.y[d]);
                row_shift = d * scatter.rows_per_dst;
            }
            const bool last = tile + num_pairs >= tiles_total;
            store_columns<OutT, kCols, ADD>(acc, (store_flags & 4) && last ? smem + ew * kBlocks<OutT, kCols>() * 4096 : nullptr, my_store, colw + col0,
                                       colb + col0, map_o, map_t, outp, ldo, row_shift, row_base, Q, n0 + col0, R, scale_inv, has_bias, relu,
                                       fin, store_flags);
        }
        if constexpr (REQ) {
            __syncwarp();
            cluster_arrive();
        }
        if (elect_one()) tma_store_wait_read();    // shared memory is read until then
    }

    if (threadIdx.x == 0 && *abort_flag) {
        // Error path only: give copies that are still in flight time to land before the smem goes away.
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {}
    }
    tc_fence_before();
    __syncthreads();
    // The peer may still be reading this CTA's shared memory or arriving on its barriers: every warp has arrived as soon as it
    // was done with the other CTAs' memory, the epilogue's before their last stores.
    cluster_wait();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem_base), "r"(static_cast<uint32_t>(C::kTmemCols)) : "memory");
    }
}

}  // namespace pair
