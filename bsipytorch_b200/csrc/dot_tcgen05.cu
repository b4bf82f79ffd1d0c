// Dot core on the 5th-generation tensor cores.
//
// The 7 query slices and 6 key slices are recombined into signed 8-bit operands, so that the
// per-chunk integer accumulator
//     I[q][r][c] = sum_{d in chunk c} a8[q][d] * k8[r][d]
// (identical to sum_{i,j} +-2^(i+j) popc(A_i & B_j), the reference's weighted popcount,
// bsi_cuda_kernels_dot.cuh:1447-1517) is ONE int8 contraction of depth 256 instead of 42
// binary MMAs. Per output tile of 128 query rows x BN key rows:
//
//   warp 0   TMA producer: per 128-byte k-block, one box of A (128 x 128 B) and one of B
//            (BN x 128 B), 128-byte swizzled, into a ring of smem stages (mbarrier full/empty)
//   warp 1   MMA issuer: per chunk 2 k-blocks x 4 tcgen05.mma.kind::i8 (M=128, N=BN, K=32) into one
//            of two TMEM accumulators (int32, BN columns each); tcgen05.commit frees the stage
//            and, after the 8th MMA, publishes the accumulator
//   warps 2+ epilogue: tcgen05.ld the finished accumulator, acc = fmaf(float(I), qs[q][c], acc)
//            in registers, in chunk order (the reference's order, :1519-1526), hand the TMEM
//            buffer back; at the end out = acc * bw0[r] * scale_inv.
//
// The chunk scale cannot ride inside the integer contraction (each chunk has its own power of
// two per row), which is why the accumulator is drained every 256 of depth; the two TMEM buffers
// let the drain of chunk c overlap the MMAs of chunk c+1.
//
// Every wait is bounded: on a timeout the waiting role records a site code in a device status
// word, raises a CTA-wide abort flag, every role leaves its loop, outstanding copies and MMAs
// are waited for (bounded again), TMEM is freed and the kernel returns.
#include <cuda.h>
#include <stdlib.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "epilogue.cuh"
#include "quantise.cuh"

namespace bsi {

// Device-side status word: 0 = clean; otherwise the site code of the first wait that gave up.
__device__ int g_device_status = 0;
// warp-tiles of the paired kernel that took the integer accumulation (a test hook: bsi_b200_debug_exact_int_tiles)
__device__ unsigned long long g_exact_int_tiles = 0ull;

namespace {

constexpr int BM = 128;     // query rows per tile = TMEM lanes
constexpr int BK = 128;     // int8 per k-block = one 128-byte swizzle row
constexpr int UMMA_K = 32;  // depth of one kind::i8 instruction
constexpr int kEpiWarps = 8;
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr long long kWaitCycles = 4000000000ll;  // ~2 s at B200 clocks; real waits are microseconds

enum Site { kSiteProducer = 1, kSiteMmaFull = 2, kSiteMmaTmem = 3, kSiteEpilogue = 4, kSiteDrain = 5 };

template <int BN>
struct Cfg {
    static constexpr int kStages = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
    static constexpr int kABytes = BM * BK;
    static constexpr int kBBytes = BN * BK;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kTmemCols = 2 * BN;  // two accumulators; 128, 256 or 512: powers of two
    static constexpr int kBarriers = 2 * kStages + 5;
    static constexpr int kSmemBytes = kStages * kStageBytes + kBarriers * 8 + 16 + 1024;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// try_wait that lets the hardware park the thread for up to `hint_ns` before it reports "not yet":
// a parked thread issues nothing, so waiting warps do not steal issue slots from the MMA issuer.
__device__ __forceinline__ bool mbar_try_parked(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}

// Bounded wait. Returns false when the CTA is aborting (this wait or another one timed out).
// The abort flag and the clock are looked at only every 16th unsuccessful (parked) try.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int site) {
    if (mbar_try(bar, parity)) return true;
    long long t0 = 0;
    for (uint32_t spins = 1;; ++spins) {
        if (mbar_try_parked(bar, parity, 20000u)) return true;
        if ((spins & 15u) == 0u) {
            if (*abort_flag) return false;
            const long long now = clock64();
            if (t0 == 0) t0 = now;
            if (now - t0 > kWaitCycles) {
                *abort_flag = 1;
                atomicCAS(&g_device_status, 0, site);
                return false;
            }
        }
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// K-major, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart (SBO), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1024u >> 4) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

// kind::i8: D = S32 (2 at bit 4), A and B signed 8-bit (1 at bits 7 and 10), both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t umma_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(BM >> 4) << 24);
}

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, int32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// 16 columns into r[0..15] (the tail piece of tiles whose column count per warp is not a multiple of 32).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// The same with the registers of the load named, so that nothing touches them before: for loads under way beside other work.
__device__ __forceinline__ void tmem_ld_wait_for(int32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]),
                   "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

template <int BN, bool DBG>
__global__ void __launch_bounds__(kThreads, 1) dot_i8_tcgen05_kernel(
    const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
    const float* __restrict__ qs, int64_t qs_stride, const float* __restrict__ bw0,
    int Q, int R, int chunks, float scale_inv, float* __restrict__ out, int64_t ldo,
    int32_t* __restrict__ dbg_iacc) {
    using C = Cfg<BN>;
    constexpr int kStages = C::kStages;
    constexpr int kCols = BN / 2;  // accumulator columns per epilogue warp

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * C::kStageBytes);
    // bars: full[kStages], empty[kStages], tfull[2], tempty[2], drain
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kBarriers);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
    auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * kStages + b); };
    auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * kStages + 2 + b); };
    const uint32_t drain_bar = bar_base + 8u * (2 * kStages + 4);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BN;
    const int m0 = blockIdx.y * BM;
    const int num_kb = chunks * 2;

    if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), kEpiWarps * 32);
        }
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(static_cast<uint32_t>(C::kTmemCols)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int kb = 0; kb < num_kb; ++kb) {
                const int s = kb % kStages;
                const uint32_t ph = static_cast<uint32_t>(kb / kStages) & 1u;
                if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, kSiteProducer)) break;
                mbar_expect_tx(full_bar(s), C::kStageBytes);
                const uint32_t a_dst = smem_base + s * C::kStageBytes;
                tma_load_2d(a_dst, &map_a, kb * BK, m0, full_bar(s));
                tma_load_2d(a_dst + C::kABytes, &map_b, kb * BK, n0, full_bar(s));
                issued = kb + 1;
            }
            if (*abort_flag) {
                // Let every copy that was issued land before the CTA gives its smem back.
                const int first = issued > kStages ? issued - kStages : 0;
                for (int kb = first; kb < issued; ++kb) {
                    const int s = kb % kStages;
                    const uint32_t ph = static_cast<uint32_t>(kb / kStages) & 1u;
                    const long long t0 = clock64();
                    while (!mbar_try(full_bar(s), ph) && clock64() - t0 < kWaitCycles / 64) {}
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc(BN);
            bool ok = true;
            for (int c = 0; c < chunks && ok; ++c) {
                const int b = c & 1;
                const uint32_t tph = static_cast<uint32_t>(c >> 1) & 1u;
                if (!mbar_wait(tempty_bar(b), tph ^ 1u, abort_flag, kSiteMmaTmem)) { ok = false; break; }
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(b * BN);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int kb = 2 * c + half;
                    const int s = kb % kStages;
                    const uint32_t ph = static_cast<uint32_t>(kb / kStages) & 1u;
                    if (!mbar_wait(full_bar(s), ph, abort_flag, kSiteMmaFull)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_base + s * C::kStageBytes;
                    const uint64_t adesc = umma_desc(a_addr);
                    const uint64_t bdesc = umma_desc(a_addr + C::kABytes);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        // +32 bytes of K inside the swizzle row = +2 in the 16-byte address field
                        umma_i8(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc, (half | k) != 0 ? 1u : 0u);
                    }
                    umma_commit(empty_bar(s));
                }
                if (ok) umma_commit(tfull_bar(b));
            }
            if (!ok) {
                // Wait (bounded) for whatever MMAs are still in flight before TMEM is freed.
                umma_commit(drain_bar);
                const long long t0 = clock64();
                while (!mbar_try(drain_bar, 0) && clock64() - t0 < kWaitCycles / 64) {}
            }
        }
    } else {
        const int quad = warp & 3;                 // TMEM lane quadrant this warp may read
        const int half = (warp - 2) >> 2;          // which half of the BN columns
        const int row = m0 + quad * 32 + lane;     // query row of this thread
        const int col0 = half * kCols;
        const bool row_ok = row < Q;
        const float* qs_row = qs + static_cast<int64_t>(row_ok ? row : 0) * (qs_stride ? qs_stride : 1);
        float acc[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j) acc[j] = 0.0f;

        bool ok = true;
        for (int c = 0; c < chunks && ok; ++c) {
            const int b = c & 1;
            const uint32_t tph = static_cast<uint32_t>(c >> 1) & 1u;
            const float qscale = qs_stride ? __ldg(qs_row + c) : __ldg(qs_row);
            if (!mbar_wait(tfull_bar(b), tph, abort_flag, kSiteEpilogue)) { ok = false; break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) +
                                   static_cast<uint32_t>(b * BN + col0);
#pragma unroll
            for (int j = 0; j < kCols / 32; ++j) {
                int32_t v[32];
                tmem_ld32(taddr + j * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    acc[j * 32 + e] = __fmaf_rn(static_cast<float>(v[e]), qscale, acc[j * 32 + e]);
                }
                if (DBG) {
                    if (row_ok) {
#pragma unroll
                        for (int e = 0; e < 32; ++e) {
                            const int col = n0 + col0 + j * 32 + e;
                            if (col < R)
                                dbg_iacc[(static_cast<int64_t>(row) * R + col) * chunks + c] = v[e];
                        }
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(tempty_bar(b));
        }
        if (ok && row_ok) {
            float* orow = out + static_cast<int64_t>(row) * ldo;
            const bool vec = ((reinterpret_cast<uintptr_t>(orow) & 15) == 0) &&
                             ((reinterpret_cast<uintptr_t>(bw0) & 15) == 0) && (n0 + col0 + kCols <= R);
            if (vec) {
#pragma unroll
                for (int j = 0; j < kCols; j += 4) {
                    const int col = n0 + col0 + j;
                    const float4 w = __ldg(reinterpret_cast<const float4*>(bw0 + col));
                    float4 o;
                    o.x = (acc[j + 0] * w.x) * scale_inv;
                    o.y = (acc[j + 1] * w.y) * scale_inv;
                    o.z = (acc[j + 2] * w.z) * scale_inv;
                    o.w = (acc[j + 3] * w.w) * scale_inv;
                    *reinterpret_cast<float4*>(orow + col) = o;
                }
            } else {
#pragma unroll
                for (int j = 0; j < kCols; ++j) {
                    const int col = n0 + col0 + j;
                    if (col < R) orow[col] = (acc[j] * __ldg(bw0 + col)) * scale_inv;
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem_base), "r"(static_cast<uint32_t>(C::kTmemCols)) : "memory");
    }
}

#include "dot_tcgen05_pair.cuh"
#include "dot_rows_tcgen05.cuh"

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &qres) ==
                cudaSuccess && qres == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
        }
    }
    return fn;
}

// [rows, depth] int8, row stride ld bytes; box = 128 bytes of depth x box_rows rows, 128-byte
// swizzle; rows beyond `rows` read as zero.
int make_map(CUtensorMap* map, const int8_t* base, int64_t rows, int64_t depth, int64_t ld, int box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return fail(BSI_ERR_CUDA, "dot_i8: cuTensorMapEncodeTiled entry point not found");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(depth), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(BK), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<int8_t*>(base), dims, strides, box,
                          estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("dot_i8: cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
        return BSI_ERR_CUDA;
    }
    return BSI_OK;
}

// The output as destination of bulk stores: [rows, cols] elements of esz bytes, boxes of 32 rows x box_bytes, whose
// 16-byte pieces are swizzled by row (128- or 64-byte rows).
int make_out_map(CUtensorMap* map, void* out, int esz, int64_t rows, int64_t cols, int64_t ld, int box_bytes) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return fail(BSI_ERR_CUDA, "dot_i8: cuTensorMapEncodeTiled entry point not found");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld * esz)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_bytes / esz), 32u};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, esz == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, out, dims, strides,
                          box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                          CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("dot_i8: cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
        return BSI_ERR_CUDA;
    }
    return BSI_OK;
}

template <int BN, bool DBG>
int launch_tile(const CUtensorMap& ma, const CUtensorMap& mb, const float* qs, int64_t qs_stride,
                const float* bw0, int Q, int R, int chunks, float scale_inv, float* out, int64_t ldo,
                int32_t* dbg, cudaStream_t stream) {
    using C = Cfg<BN>;
    static bool attr_set[64] = {false};
    int dev = 0;
    BSI_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        BSI_CUDA_TRY(cudaFuncSetAttribute(dot_i8_tcgen05_kernel<BN, DBG>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    dim3 grid((R + BN - 1) / BN, (Q + BM - 1) / BM, 1);
    dot_i8_tcgen05_kernel<BN, DBG><<<grid, kThreads, C::kSmemBytes, stream>>>(
        ma, mb, qs, qs_stride, bw0, Q, R, chunks, scale_inv, out, ldo, dbg);
    return check_launch("dot_i8 tcgen05 launch");
}

// How many clusters of 2 * SPLIT CTAs run at once (one CTA per SM whatever the instantiation); 0 when the query fails.
template <int SPLIT>
int resident_clusters();

template <int BN, bool DBG, typename OutT, bool REQ = false, int SPLIT = 1, bool ADD = false, bool ONE = false>
int launch_pair(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mo, const CUtensorMap& mt, int vector_store,
                const float* qs, int64_t qs_stride, const float* bw0, const float* bias, int Q, int R, int chunks,
                float scale_inv, void* out, int64_t ldo, int32_t* dbg, const ScatterDst& scatter,
                const RequantDst& requant, const Finishing& fin, const float* k_abs_sum, float q_abs_max, const float* q_sq, int64_t q_sq_stride,
                cudaStream_t stream, int* max_clusters_out = nullptr /* only asks how many clusters fit at once */) {
    using C = pair::Cfg<BN, OutT, REQ, SPLIT>;
    static bool attr_set[64] = {false};   // per instantiation
    int dev = 0;
    BSI_CUDA_TRY(cudaGetDevice(&dev));
    const int tiles_m = (Q + 255) / 256;
    const int tiles_n = (R + BN - 1) / BN;
    const int tiles_total = tiles_m * tiles_n;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * SPLIT;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // programmatic dependent launch: this kernel's set-up may overlap the tail of the kernel before it
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(pair::kThreads, 1, 1);
    cfg.dynamicSmemBytes = C::kSmemBytes;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        BSI_CUDA_TRY(cudaFuncSetAttribute(pair::dot_i8_tcgen05_pair_kernel<BN, DBG, OutT, REQ, SPLIT, ADD, ONE>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    if (max_clusters_out != nullptr) {
        cfg.gridDim = dim3(2 * SPLIT * (sm_count() / (2 * SPLIT)), 1, 1);
        BSI_CUDA_TRY(cudaOccupancyMaxActiveClusters(max_clusters_out, pair::dot_i8_tcgen05_pair_kernel<BN, DBG, OutT, REQ, SPLIT, ADD, ONE>, &cfg));
        return BSI_OK;
    }
    int clusters = tiles_total;
    if constexpr (SPLIT == 1 && !ONE) {
        const int resident = resident_clusters<1>();
        if (resident <= 0) return fail(BSI_ERR_CUDA, "dot_i8: no cluster of 2 CTAs fits on this device");
        clusters = tiles_total < resident ? tiles_total : resident;
    }
    cfg.gridDim = dim3(2 * SPLIT * clusters, 1, 1);
    BSI_CUDA_TRY(cudaLaunchKernelEx(&cfg, pair::dot_i8_tcgen05_pair_kernel<BN, DBG, OutT, REQ, SPLIT, ADD, ONE>, ma, mb, mo, mt, vector_store, qs,
                                    qs_stride, bw0, bias, Q, R, chunks, tiles_m, tiles_total, scale_inv, out, ldo, dbg, scatter, requant,
                                    fin, k_abs_sum, q_abs_max, q_sq, q_sq_stride));
    return check_launch("dot_i8 tcgen05 pair launch");
}

// Pair kernel tile width. The costs, 650 + 3.1 * BN cycles per 256-deep chunk of a tile and ceil(tiles / pairs) tiles, and those of
// pick_split were fitted to a form of the kernel whose chunks took 980 cycles at every width; they take 500 + 2 * BN now. Over 228
// sizes (64 .. 2048 rows, 256 .. 12288 columns, 2 .. 64 chunks) what the two pick is within 1.1 % of the best width and split on
// the mean, a refitted rule within 0.3 %; the difference is at 8192 and more of depth, where unsplit tiles of 64 to 128 columns
// are 6 to 25 % shorter than the split taken (512 x 3072 x 16384: 32.4 us, 96 columns 26.0). The widest tile wins unless a narrower one is clearly cheaper (more than 8 %: at equal
// rounds the wider tile also has the shorter fill and store phases). float32 output may use any multiple of 32,
// the 16-bit layer epilogues (whole 64-column store rounds) the powers of two.
int pick_bn_pair(int64_t Q, int64_t R, bool any_width) {
    const int pairs = sm_count() / 2;
    const int64_t mt = (Q + 255) / 256;
    int best = 256;
    double best_cost = 1e300;
    for (int bn = 256; bn >= 64; bn -= 32) {
        if (!any_width && bn != 256 && bn != 128 && bn != 64) continue;
        const int64_t tiles = mt * ((R + bn - 1) / bn);
        const int64_t waves = (tiles + pairs - 1) / pairs;
        const double cost = static_cast<double>(waves) * (650.0 + 3.1 * bn);
        if (cost < best_cost * 0.92) {
            best_cost = cost;
            best = bn;
        }
    }
    return best;
}

// Tile width and parts along K of this thread's last paired dot (a test hook: bsi_b200_debug_last_tiles).
thread_local int t_last_width = 0, t_last_parts = 0;

template <int SPLIT>
int resident_clusters() {
    static int cached[64] = {0};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (cached[dev] == 0) {
        const CUtensorMap none = {};
        if (launch_pair<64, false, float, false, SPLIT>(none, none, none, none, 0, nullptr, 0, nullptr, nullptr, 0, 0, 1, 0.0f, nullptr, 0,
                                                        nullptr, ScatterDst{}, RequantDst{}, Finishing{}, nullptr, 0.0f, nullptr, 0, nullptr, &n) != BSI_OK)
            n = 0;
        cached[dev] = n > 0 ? n : -1;
    }
    return cached[dev] > 0 ? cached[dev] : 0;
}

// Split along K or not, and the tile width to split at: *bn and the number of parts, 1 for no split. The costs are cycles
// fitted to runs of 2 .. 64 chunks at widths 64, 128 and 256: 820 + 1.3 bn per chunk, and beside the chunks 7000 + 25 bn
// without a split, 7500 + 55 bn with two parts, 12000 + 47 bn with four (clusters of eight start later). A split takes one
// wave of clusters (33 of four CTAs and 15 of eight fit) and has to save a fifteenth. *cycles: the cost of what is split.
// sums: the queries' sums of squares are there, so that the vote passes but for rare rows. Without them it rests on the two
// cheap bounds, which hold for even activations and mostly fail for layer norms' outputs with outliers, and a tile whose vote fails
// is done by one pair after all: a wager on the values. Taken where it wins at least about as much as it may lose (40 .. 512 rows,
// 256 .. 4096 columns, float16, split over unsplit): tiles of the unsplit width, four parts from 24 chunks on, 0.53 .. 0.84 where
// the vote passes and 1.21 .. 1.29 where it fails (64 x 512 x 16384: 10.4 and 25.6 us, unsplit 18.1 and 21.0), two from 48 on,
// 0.75 .. 0.86 and 1.18 .. 1.22. Not taken: two parts below (32 chunks 0.84 .. 0.92 and 1.22 .. 1.25), wider tiles than unsplit (0.72 ..
// 1.23 and 1.60 .. 1.90: 512 x 8192 -> 2048 13.3 and 21.5, unsplit 12.0 and 12.8).
int pick_split(int64_t Q, int64_t R, int64_t chunks, int unsplit_bn, bool sums, int* bn, double* cycles) {
    const int64_t mt = (Q + 255) / 256, pairs = sm_count() / 2;
    if (mt * ((R + unsplit_bn - 1) / unsplit_bn) > pairs) return 1;
    auto cost = [&](int w, double fixed, double per_column, int64_t parts) {
        return fixed + per_column * w + static_cast<double>((chunks + parts - 1) / parts) * (820.0 + 1.3 * w);
    };
    double best = 0.93 * cost(unsplit_bn, 7000.0, 25.0, 1);
    int parts = 1;
    if (cost(64, 7500.0, 55.0, 4) >= best) return 1;       // not even the cheapest one: no need to ask the driver
    for (int s = 2; s <= 4; s *= 2) {
        const int64_t room = s == 2 ? resident_clusters<2>() : resident_clusters<4>();
        for (int w = 256; w >= 64; w /= 2) {
            if (mt * ((R + w - 1) / w) > room) continue;
            if (!sums && (w != unsplit_bn || chunks < (s == 4 ? 24 : 48))) continue;
            const double c = s == 2 ? cost(w, 7500.0, 55.0, 2) : cost(w, 12000.0, 47.0, 4);
            if (c < best) {
                best = *cycles = c;
                parts = s;
                *bn = w;
            }
        }
    }
    return parts;
}

// ---- dots of few rows (dot_rows_tcgen05.cuh) ------------------------------------------------------------------------
struct RowsPlan {
    int nq, parts, per_part, stages, bufs;
    double us;       // what the launch is expected to take (fused form)
};

// Query tile, CTAs along K, ring sizes; false where the kernel has no form for the size. The costs are microseconds fitted
// to layers of 1 .. 32 chunks on an idle GPU: a chunk of 16 rows to quantise 0.62, of 32 rows 1.2, the key stream alone 0.36,
// and for every part behind the first the hand-over and the folding of its chunks.
bool plan_rows(int64_t Q, int64_t R, int64_t chunks, bool fused, RowsPlan* out) {
    const int sms = sm_count();
    RowsPlan best = {};
    best.us = 1e30;
    for (int nq = 16; nq <= 32; nq *= 2) {
        if (!fused && (nq < Q || (nq == 32 && Q <= 16))) continue;
        const int64_t tiles = ((R + 127) / 128) * ((Q + nq - 1) / nq);
        for (int s = 1; s <= 8; s *= 2) {
            const int64_t per = (chunks + s - 1) / s, parts = (chunks + per - 1) / per;
            // a split runs in one wave and keeps all of its accumulators; so does the fused form, whose tiles quantise alone
            // (of 148 SMs, clusters of four use 132 at once and clusters of eight 120)
            if ((s > 1 || fused) && tiles * parts > (s <= 2 ? sms : s == 4 ? sms * 9 / 10 : sms * 5 / 6)) break;
            if (s > 1 && (parts == 1 || per > rows::kMaxBufs || per * nq > rows::kTmemCols)) continue;
            const double rows_of_tile = static_cast<double>(std::min<int64_t>(Q, nq));
            RowsPlan p = {};
            if (!fused) p.us = 0.36 * per + (parts - 1) * (0.7 + 0.12 * per);
            else if (nq == 16) p.us = 3.0 + (0.33 + 0.018 * rows_of_tile) * per + (parts - 1) * (0.6 + 0.15 * per);
            else p.us = 3.9 + 1.2 * per + (parts - 1) * (0.8 + 0.25 * per);
            if (p.us >= best.us) continue;
            p.nq = nq;
            p.parts = static_cast<int>(parts);
            p.per_part = static_cast<int>(per);
            const int64_t left = rows::kSmemBytes - rows::kFixedBytes - (parts > 1 ? rows::kEpiWarps * nq * 128 : 0) - per * nq * 4;
            p.stages = static_cast<int>(std::min<int64_t>(std::min<int64_t>(rows::kMaxStages, per), left / (rows::kABytes + nq * 2 * BK)));
            p.bufs = parts > 1 ? p.per_part : p.stages;
            if (left > 0 && p.stages >= std::min<int64_t>(per, 2)) best = p;
        }
    }
    *out = best;
    return best.us < 1e30;
}

// Rows kernels this thread has launched since it last asked, and the last one's plan (a test hook: bsi_b200_debug_last_rows).
thread_local int t_rows_launches = 0;
thread_local RowsPlan t_last_rows = {};

template <int NQ, typename OutT, typename XT>
int launch_rows(const CUtensorMap& mk, const CUtensorMap& mq, const RowsPlan& plan, const rows::Args& a, cudaStream_t stream) {
    static bool attr_set[64] = {false};
    int dev = 0;
    BSI_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        BSI_CUDA_TRY(cudaFuncSetAttribute(rows::dot_rows_kernel<NQ, OutT, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows::kSmemBytes));
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    constexpr bool kFuse = !std::is_same<XT, void>::value;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (plan.parts > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = static_cast<unsigned>(plan.parts);
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.gridDim = dim3(static_cast<unsigned>((a.R + 127) / 128 * plan.parts), static_cast<unsigned>((a.Q + NQ - 1) / NQ), 1);
    cfg.blockDim = dim3((2 + rows::kEpiWarps + (kFuse ? rows::kQuantWarps : 0)) * 32, 1, 1);
    cfg.dynamicSmemBytes = rows::kSmemBytes;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = n;
    BSI_CUDA_TRY(cudaLaunchKernelEx(&cfg, rows::dot_rows_kernel<NQ, OutT, XT>, mk, mq, a));
    return check_launch("dot_i8 rows launch");
}

// a8: the packed queries, null in the fused form (whose activations are in `a`).
int run_rows(const RowsPlan& plan, rows::Args a, const int8_t* a8, int64_t lda, const int8_t* k8, int64_t ldk, int x_dtype, int y_dtype,
             cudaStream_t stream) {
    a.parts = plan.parts; a.per_part = plan.per_part; a.stages = plan.stages; a.bufs = plan.bufs;
    CUtensorMap mk, mq = {};
    if (int rc = make_map(&mk, k8, a.R, static_cast<int64_t>(a.chunks) * 256, ldk, 128)) return rc;
    if (a8 != nullptr)
        if (int rc = make_map(&mq, a8, a.Q, static_cast<int64_t>(a.chunks) * 256, lda, plan.nq)) return rc;
    ++t_rows_launches;
    t_last_rows = plan;
#define BSI_ROWS(O_, X_) (plan.nq == 16 ? launch_rows<16, O_, X_>(mk, mq, plan, a, stream) : launch_rows<32, O_, X_>(mk, mq, plan, a, stream))
    if (a8 == nullptr)
        return x_dtype == BSI_DTYPE_F32 ? BSI_ROWS(float, float) : x_dtype == BSI_DTYPE_F16 ? BSI_ROWS(__half, __half) : BSI_ROWS(__nv_bfloat16, __nv_bfloat16);
    return y_dtype == BSI_DTYPE_F32 ? BSI_ROWS(float, void) : y_dtype == BSI_DTYPE_F16 ? BSI_ROWS(__half, void) : BSI_ROWS(__nv_bfloat16, void);
#undef BSI_ROWS
}

}  // namespace

// Whether the paired tiles, split along K, are the shorter way for 17 to 32 rows: with few key tiles and a deep K, where the
// rows kernel's parts hand their sums on one after another and the split adds all parts at once (16384 x 512, 32 rows: 15.4 us
// against 19.1; 8192 x 512: 11.1 against 12.5; 6144 x 512: 10.2 against 10.8; the other way 8192 x 1024: 13.5 against 12.5, 4096
// x 512: 8.5 against 8.6). Only where its bounds are given and quickly read (rows of whole 16-byte vectors): without them the
// split does not happen or starts late (4608 x 4608: 21.9 us against 9.5). Both costs as above, in microseconds of a replayed
// graph: beside its chunks and hand-overs the rows kernel takes 2.1 + 0.2 per part + 0.045 per row, a split (1900 cycles to
// the microsecond) 0.1 less for every tile that a wave of clusters of eight would still have room for. Split and rows kernel as they
// were when this was fitted; both have become shorter (512 keys 15.4 -> 10.5 us, 1024 keys on the rows kernel 17.0 -> 13.2).
static bool split_is_shorter(int64_t Q, int64_t R, int64_t chunks, const RowsPlan& rows_plan, const bsi_dot_bounds& bounds, int64_t qs_stride) {
    if (rows_plan.parts == 1 || bounds.key_bounds == nullptr || bounds.query_sq == nullptr || qs_stride < chunks ||
        bounds.query_sq_stride < chunks || ((chunks | qs_stride | bounds.query_sq_stride) & 3) != 0)
        return false;
    int bn = pick_bn_pair(Q, R, false);
    double cycles = 0.0;
    if (pick_split(Q, R, chunks, bn, true, &bn, &cycles) == 1) return false;
    const double split_us = cycles / 1900.0 - 0.1 * static_cast<double>(15 - (R + bn - 1) / bn);
    return split_us < rows_plan.us + 2.1 + 0.2 * rows_plan.parts + 0.045 * static_cast<double>(Q);
}

double decode_share(int64_t Q, int64_t chunks);

// Up to 16 rows and more key tiles than SMs: the rows kernel starts another wave of CTAs, each with its set-up and nothing beside
// it on the SM, and a wave that is not full takes its SMs' time all the same, where the key-streaming kernel goes on. It pays
// where that kernel leaves a quarter of its warps without a chunk (5 chunks: 20480 x 1280, 1 row, 8.2 -> 7.5 us; 10 chunks: 33664 x
// 2560, 16 rows, 25.9 -> 18.5) or where long waves are nearly full (37888 x 4096, 1 row, 29.4 -> 26.0, 30000 x 4096, 16 rows,
// 26.7 -> 25.4; 8192 deep from three quarters on, 30000 rows 42.9 -> 40.6, and beyond 8 rows whatever the fill, 26000 rows 46.2
// -> 41.6). It loses elsewhere: 19072 x 4096, 1 row, 16.4 us against 19.2; 50272 x 768, 8 rows, 10.9 against 13.2; 50272 x
// 2048, 1 row, 19.4 against 20.4.
static bool more_waves_pay(int64_t Q, int64_t R, int64_t chunks) {
    const int64_t tiles = (R + 127) / 128, sms = sm_count(), waves = (tiles + sms - 1) / sms;
    if (waves == 1) return true;
    const double fill = static_cast<double>(tiles) / static_cast<double>(waves * sms);
    if (chunks >= 5 && decode_share(Q, chunks) <= 0.75) return true;
    const double least = chunks >= 24 ? (Q > 8 ? 0.0 : 0.75) : chunks >= 14 ? (Q > 8 ? 0.75 : 0.85) : 2.0;
    return fill >= least;
}

// Whether a dot of packed queries goes to the rows kernel. 17 to 32 rows, which fill an eighth of a paired tile: but for the
// case above (4096 x 16384 float16 layers of 32 rows 20.3 -> 17.5 us, 8192 x 2048 18.2 -> 15.1). Up to 16, where the
// key-streaming kernel is the other choice: with key tiles for most of the SMs (4096 x 16384, 16 rows: 19.3 -> 16.0 us; 4096 x
// 11008, 8 rows: 13.5 -> 11.6) and, beyond 8 rows, which that kernel's MMAs are too slow for, from 48 MB of keys on (16384 x
// 4096: 28.6 -> 24.1); smaller sets it spreads better (8192 x 2048, 16 rows: 11.5 us against 12.5), and most
// sets of more than one wave too (above).
bool rows_fits(int64_t Q, int64_t R, int64_t chunks, const bsi_dot_bounds& bounds, int64_t qs_stride) {
    if (Q > 32 || R >= (1 << 24) || chunks >= (1 << 12)) return false;
    RowsPlan plan;
    if (Q > 16) return plan_rows(Q, R, chunks, false, &plan) && !split_is_shorter(Q, R, chunks, plan, bounds, qs_stride);
    return (R >= 10240 || (Q > 8 && R * chunks * 256 >= (48 << 20))) && more_waves_pay(Q, R, chunks) && plan_rows(Q, R, chunks, false, &plan);
}

int dot_rows(const int8_t* a8, int64_t lda, const float* qs, int64_t qs_stride, const int8_t* k8, int64_t ldk, const float* bw0,
             const float* bias, int64_t Q, int64_t R, int64_t chunks, float scale_inv, void* out, int64_t ldo, int y_dtype,
             const Finishing& fin, bool keys_complete, cudaStream_t stream) {
    RowsPlan plan;
    if (!plan_rows(Q, R, chunks, false, &plan)) return fail(BSI_ERR_UNSUPPORTED, "dot_i8: no rows form for these sizes");
    rows::Args a = {};
    a.qs = qs; a.qs_stride = qs_stride; a.bw0 = bw0; a.bias = bias; a.keys_complete = keys_complete ? 1 : 0;
    a.Q = static_cast<int>(Q); a.R = static_cast<int>(R); a.chunks = static_cast<int>(chunks);
    a.scale_inv = scale_inv; a.out = out; a.ldo = ldo; a.fin = fin;
    return run_rows(plan, a, a8, lda, k8, ldk, 0, y_dtype, stream);
}

// Paired-CTA engine with the output type and the bias chosen at run time (y_dtype: BSI_DTYPE_*).
int dot_i8_pair(const int8_t* a8, int64_t lda, const float* qs, int64_t qs_stride, const int8_t* k8, int64_t ldk,
                const float* bw0, const float* bias, int64_t Q, int64_t R, int64_t chunks, float scale_inv,
                void* out, int64_t ldo, int y_dtype, int32_t* dbg_iacc, int force_bn, const Finishing& fin,
                const ScatterDst* scatter_in, const RequantDst* requant_in, const bsi_dot_bounds& bounds, cudaStream_t stream) {
    RequantDst requant = {};
    if (requant_in != nullptr) {
        requant = *requant_in;
        if (requant.n < 1 || requant.n > BSI_B200_MAX_PEERS || (R & 255) != 0 ||
            (y_dtype != BSI_DTYPE_F16 && y_dtype != BSI_DTYPE_BF16) || dbg_iacc != nullptr || scatter_in != nullptr)
            return fail(BSI_ERR_INVALID, "dot_i8: re-quantised output needs R % 256 == 0 and a 16-bit layer type");
        force_bn = 256;   // one tile row = one 256-column chunk
    }
    ScatterDst scatter = {};
    if (scatter_in != nullptr) {
        scatter = *scatter_in;
        if (scatter.n < 1 || scatter.n > BSI_B200_MAX_PEERS || scatter.rows_per_dst <= 0 || (scatter.rows_per_dst & 31) != 0 ||
            static_cast<int64_t>(scatter.n) * scatter.rows_per_dst < Q)
            return fail(BSI_ERR_INVALID, "dot_i8: scatter needs 1..16 destinations of a multiple of 32 rows covering Q");
        out = scatter.y[0];
    }
    if (Q > 0x7fffff00ll || R > 0x7fffff00ll || chunks > 0x400000)
        return fail(BSI_ERR_UNSUPPORTED, "dot_i8: Q, R or chunks too large");
    const bool any_width = y_dtype == BSI_DTYPE_F32 && fin.add == nullptr;      // sums are built for the powers of two
    // bounds of the two images switch on the integer accumulation where it is provably exact
    const float* kabs = bounds.key_bounds;
    const float qabs = static_cast<float>(bounds.query_abs_max);
    const bool has_sq = kabs != nullptr && qs_stride != 0 && bounds.query_sq_stride >= chunks;
    const float* qsq = has_sq ? bounds.query_sq : nullptr;
    const int64_t qsq_stride = bounds.query_sq_stride;
    int bn = force_bn ? force_bn : pick_bn_pair(Q, R, any_width);
    if (!force_bn && any_width && bn == 256 && kabs != nullptr && qsq != nullptr) {
        // Both sides carry their bounds, so the integer route is likely, and with its cheaper epilogue a single
        // wave of 256 x 224 tiles on more pairs beats one of 256 x 256 tiles (measured on 512 x 8192 x 2048:
        // 13.64 against 13.82 us; with the float32 chain the two are even).
        const int64_t pairs = sm_count() / 2, mt = (Q + 255) / 256;
        const int64_t t256 = mt * ((R + 255) / 256), t224 = mt * ((R + 223) / 224);
        if (t256 <= pairs && t224 <= pairs && t224 > t256) bn = 224;
    }
    // only with bounds (a split adds integers), one plain destination, and no accumulator dump
    const bool may_split = !force_bn && kabs != nullptr && dbg_iacc == nullptr && scatter.n == 0;
    double cycles = 0.0;
    const int parts = may_split ? pick_split(Q, R, chunks, bn, qsq != nullptr || qs_stride == 0, &bn, &cycles) : 1;
    t_last_width = bn;
    t_last_parts = parts;
    if (bn < 64 || bn > 256 || (bn & 31) != 0 || (!any_width && (bn & (bn - 1)) != 0))
        return fail(BSI_ERR_INVALID, "dot_i8: tile width must be a multiple of 32 in [64, 256] (64, 128 or 256 for 16-bit outputs)");
    if (dbg_iacc != nullptr && y_dtype != BSI_DTYPE_F32)
        return fail(BSI_ERR_INVALID, "dot_i8: the accumulator dump is only available with float32 output");
    CUtensorMap ma, mb;
    if (int rc = make_map(&ma, a8, Q, chunks * 256, lda, BM)) return rc;
    if (int rc = make_map(&mb, k8, R, chunks * 256, ldk, bn / 2)) return rc;
    // 16-byte stores need an aligned base, a row pitch that is a multiple of 16 bytes and R a multiple
    // of the values per 16 bytes; anything else takes the scalar store path
    const int esz = y_dtype == BSI_DTYPE_F32 ? 4 : 2;
    const int per16 = 16 / esz;
    const int vector_store =
        (((reinterpret_cast<uintptr_t>(out) & 15) == 0 && (ldo % per16) == 0 && (R % per16) == 0 &&
          (fin.add == nullptr || ((reinterpret_cast<uintptr_t>(fin.add) & 15) == 0 && (fin.ld_add % per16) == 0))) ? 1 : 0) |
        (fin.relu ? 2 : 0);   // the kernel's store_flags
    // bulk stores into the one output matrix; several destinations (scatter) keep plain stores
    CUtensorMap mo = {}, mt = {};
    int store_flags = vector_store;
    if ((vector_store & 1) && scatter.n == 0 && requant.n == 0 && ldo * esz < (1ll << 40)) {
        if (int rc = make_out_map(&mo, out, esz, Q, R, ldo, 128)) return rc;
        if (int rc = make_out_map(&mt, out, esz, Q, R, ldo, 64)) return rc;
        store_flags |= 4;
    }
    const int q = static_cast<int>(Q), r = static_cast<int>(R), c = static_cast<int>(chunks);
    if (parts > 1) {
#define BSI_SPLIT_T(BN_, S_, T_) (fin.add != nullptr ? BSI_SPLIT_A(BN_, S_, T_, true) : BSI_SPLIT_A(BN_, S_, T_, false))
#define BSI_SPLIT_A(BN_, S_, T_, A_)                                                                                        \
    launch_pair<BN_, false, T_, false, S_, A_>(ma, mb, mo, mt, store_flags, qs, qs_stride, bw0, bias, q, r, c, scale_inv, out, ldo, \
                                           nullptr, scatter, requant, fin, kabs, qabs, qsq, qsq_stride, stream)
#define BSI_SPLIT(BN_, S_)                                                    \
    (y_dtype == BSI_DTYPE_F16    ? BSI_SPLIT_T(BN_, S_, __half)               \
     : y_dtype == BSI_DTYPE_BF16 ? BSI_SPLIT_T(BN_, S_, __nv_bfloat16)        \
                                 : BSI_SPLIT_T(BN_, S_, float))
        if (parts == 2) return bn == 256 ? BSI_SPLIT(256, 2) : (bn == 128 ? BSI_SPLIT(128, 2) : BSI_SPLIT(64, 2));
        return bn == 256 ? BSI_SPLIT(256, 4) : (bn == 128 ? BSI_SPLIT(128, 4) : BSI_SPLIT(64, 4));
#undef BSI_SPLIT
#undef BSI_SPLIT_T
#undef BSI_SPLIT_A
    }
    // no more tiles than pairs, bulk stores: an instantiation of its own
    const bool one = (store_flags & 4) != 0 && dbg_iacc == nullptr && requant.n == 0 && (Q + 255) / 256 * ((R + bn - 1) / bn) <= resident_clusters<1>();
#define BSI_PAIR_ONE(BN_, T_, ADD_)                                                                                      \
    launch_pair<BN_, false, T_, false, 1, ADD_, true>(ma, mb, mo, mt, store_flags, qs, qs_stride, bw0, bias, q, r, c, scale_inv, out, \
                                                      ldo, nullptr, scatter, requant, fin, kabs, qabs, qsq, qsq_stride, stream)
#define BSI_PAIR_T(BN_, DBG_, T_)                                                                              \
    (one && !DBG_) ? BSI_PAIR_ONE(BN_, T_, false) :                                                            \
    launch_pair<BN_, DBG_, T_>(ma, mb, mo, mt, store_flags, qs, qs_stride, bw0, bias, q, r, c, scale_inv, out, ldo,  \
                               dbg_iacc, scatter, requant, fin, kabs, qabs, qsq, qsq_stride, stream)
#define BSI_PAIR_ADD(BN_, T_)                                                                                            \
    one ? BSI_PAIR_ONE(BN_, T_, true) :                                                                                  \
    launch_pair<BN_, false, T_, false, 1, true>(ma, mb, mo, mt, store_flags, qs, qs_stride, bw0, bias, q, r, c, scale_inv, out, \
                                                ldo, dbg_iacc, scatter, requant, fin, kabs, qabs, qsq, qsq_stride, stream)
#define BSI_PAIR(BN_)                                                                   \
    (fin.add != nullptr ? (y_dtype == BSI_DTYPE_F16 ? (BSI_PAIR_ADD(BN_, __half)) : y_dtype == BSI_DTYPE_BF16 ? (BSI_PAIR_ADD(BN_, __nv_bfloat16)) \
                                                                                               : (BSI_PAIR_ADD(BN_, float))) \
     : y_dtype == BSI_DTYPE_F16    ? (BSI_PAIR_T(BN_, false, __half))                     \
     : y_dtype == BSI_DTYPE_BF16 ? (BSI_PAIR_T(BN_, false, __nv_bfloat16))              \
     : dbg_iacc                  ? (BSI_PAIR_T(BN_, true, float))                       \
                                 : (BSI_PAIR_T(BN_, false, float)))
    if (requant.n > 0) {
        if (y_dtype == BSI_DTYPE_F16)
            return launch_pair<256, false, __half, true>(ma, mb, mo, mt, store_flags, qs, qs_stride, bw0, bias, q, r, c, scale_inv,
                                                         out, ldo, nullptr, scatter, requant, fin, kabs, qabs, qsq, qsq_stride, stream);
        return launch_pair<256, false, __nv_bfloat16, true>(ma, mb, mo, mt, store_flags, qs, qs_stride, bw0, bias, q, r, c,
                                                            scale_inv, out, ldo, nullptr, scatter, requant, fin, kabs, qabs, qsq,
                                                            qsq_stride, stream);
    }
#define BSI_PAIR_F32(BN_) (dbg_iacc ? (BSI_PAIR_T(BN_, true, float)) : (BSI_PAIR_T(BN_, false, float)))
    switch (bn) {
        case 256: return BSI_PAIR(256);
        case 224: return BSI_PAIR_F32(224);
        case 192: return BSI_PAIR_F32(192);
        case 160: return BSI_PAIR_F32(160);
        case 96: return BSI_PAIR_F32(96);
        case 128: return BSI_PAIR(128);
        default: return BSI_PAIR(64);
    }
#undef BSI_PAIR_F32
#undef BSI_PAIR
#undef BSI_PAIR_ADD
#undef BSI_PAIR_ONE
#undef BSI_PAIR_T
}

int dot_i8_tcgen05(const int8_t* a8, int64_t lda, const float* qs, int64_t qs_stride, const int8_t* k8,
                   int64_t ldk, const float* bw0, int64_t Q, int64_t R, int64_t chunks, float scale_inv,
                   float* out, int64_t ldo, int32_t* dbg_iacc, int force_bn, const bsi_dot_bounds& bounds, cudaStream_t stream) {
    if (Q > 0x7fffff00ll || R > 0x7fffff00ll || chunks > 0x400000)
        return fail(BSI_ERR_UNSUPPORTED, "dot_i8: Q, R or chunks too large");
    // force_bn: 0 = automatic; 64/128/256 = single-CTA tiles; 2064/2128/2256 = paired-CTA tiles.
    const bool want_pair = force_bn == 0 || force_bn >= 2000;
    if (want_pair) {
        return dot_i8_pair(a8, lda, qs, qs_stride, k8, ldk, bw0, nullptr, Q, R, chunks, scale_inv, out, ldo,
                           BSI_DTYPE_F32, dbg_iacc, force_bn ? force_bn - 2000 : 0, Finishing{}, nullptr, nullptr, bounds, stream);
    }
    const int bn = force_bn;
    CUtensorMap ma, mb;
    if (int rc = make_map(&ma, a8, Q, chunks * 256, lda, BM)) return rc;
    if (int rc = make_map(&mb, k8, R, chunks * 256, ldk, bn)) return rc;
    const int q = static_cast<int>(Q), r = static_cast<int>(R), c = static_cast<int>(chunks);
#define BSI_DISPATCH(BN_)                                                                              \
    (dbg_iacc ? launch_tile<BN_, true>(ma, mb, qs, qs_stride, bw0, q, r, c, scale_inv, out, ldo,      \
                                       dbg_iacc, stream)                                               \
              : launch_tile<BN_, false>(ma, mb, qs, qs_stride, bw0, q, r, c, scale_inv, out, ldo,     \
                                        nullptr, stream))
    switch (bn) {
        case 256: return BSI_DISPATCH(256);
        case 128: return BSI_DISPATCH(128);
        case 64: return BSI_DISPATCH(64);
        default: return fail(BSI_ERR_INVALID, "dot_i8: tile width must be 64, 128 or 256");
    }
#undef BSI_DISPATCH
}

}  // namespace bsi

extern "C" int bsi_b200_device_status(int* status_out) {
    using namespace bsi;
    if (status_out == nullptr) return fail(BSI_ERR_INVALID, "device_status: null pointer");
    BSI_CUDA_TRY(cudaDeviceSynchronize());
    int v = 0;
    BSI_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_device_status, sizeof(int)));
    if (v != 0) {
        const int zero = 0;
        BSI_CUDA_TRY(cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int)));
    }
    int pv = 0;
    if (int rc = take_peer_status(&pv)) return rc;
    if (v == 0) v = pv;
    *status_out = v;
    return BSI_OK;
}

// Where one launch, with the quantisation in every CTA, is the shorter way. Issued one by one, two launches take the host 10 us and
// more (a layer's call through its module), the kernel 0.5 us more than the plan says; the lines are where the two met:
//   tiles of 32 rows   17 to 32 rows always (24 x 1280 -> 16256 float32: 8.8 us against 12.6), else up to four chunks (56 x 1280 ->
//                      7808, five: 10.7 against 9.4)
//   17 rows and more   up to 10.2 us (374 x 3055 -> 739, 10.4 by the plan: 15.3 against 12.9)
//   up to 16 rows      the key-streaming kernel's own one-launch form comes first, and behind a packer that kernel or, from 10240 keys
//                      on, this one is the other way: up to 9.6 us (16 x 4352 -> 2185, 10.1: 10.7 against 10.1), up to 8.2 where
//                      the depth is no whole number of vectors (14 x 3291 -> 207, 8.7: 11.3 against 10.1), up to 10.3 from 12 MB of
//                      keys on, which the GPU needs longer than 10 us for (9 x 5104 -> 8960: 13.0 against 19.1), and not from
//                      40 MB on where the rows kernel reads packed rows (4 x 4096 -> 11000: 15.1 against 13.3)
static bool one_launch_plan(int64_t Q, int64_t R, int64_t D, bsi::RowsPlan* plan) {
    using namespace bsi;
    const int64_t chunks = (D + 255) / 256;
    if (Q < 1 || R < 1 || D < 1 || Q > (1 << 16) || R >= (1 << 24) || chunks >= (1 << 12)) return false;
    if (((R + 127) >> 7) * ((Q + 31) >> 5) > sm_count()) return false;      // more tiles than a wave has: no need to plan
    if (Q <= 16 && bsi_b200_linear_decode_fits(Q, R, D)) return false;
    if (!plan_rows(Q, R, chunks, true, plan)) return false;
    const int64_t keys = R * chunks * 256;
    if (Q <= 16) {
        if (R >= 10240 && keys >= (40 << 20)) return false;
        return plan->us <= (keys >= (12 << 20) ? 10.3 : (D & 7) != 0 ? 8.2 : 9.6);
    }
    return plan->us <= (plan->nq == 16 ? 10.2 : Q <= 32 ? 10.5 : 8.8);
}

// A replayed graph has no host cost. Up to 16 rows the key-streaming kernel behind a packer is the shorter way there (12 x 3072 x
// 768: 5.2 us against 7.5), and more than 32 rows in tiles of 32 lose to packer and paired tiles where those store whole vectors
// of 16 bits (512 x 1024 -> 1024 7.3 us against 9.2, 472 x 768 -> 640 6.8 against 8.2, 232 x 256 -> 1920 5.9 against 6.6; ragged
// columns 432 x 768 -> 660 9.0 against 8.3; float32 169 x 256 -> 2688 6.3 against 5.6, 69 x 768 -> 5504 7.2 against 7.3).
extern "C" int bsi_b200_linear_rows_ways(int64_t Q, int64_t R, int64_t D, int x_dtype) {
    bsi::RowsPlan plan;
    if (!one_launch_plan(Q, R, D, &plan)) return 0;
    const bool replayed = Q > 16 && (plan.nq == 16 || Q <= 32 || (R & 7) != 0 || x_dtype == BSI_DTYPE_F32);
    return BSI_ROWS_ISSUED | (replayed ? BSI_ROWS_REPLAYED : 0);
}

extern "C" int bsi_b200_linear_rows_fits(int64_t Q, int64_t R, int64_t D) {
    return (bsi_b200_linear_rows_ways(Q, R, D, BSI_DTYPE_F32) & BSI_ROWS_ISSUED) != 0 ? 1 : 0;
}

extern "C" int bsi_b200_linear_rows(const void* x, int x_dtype, int64_t ldx, int64_t D, int decimal_places, int bits, const int8_t* k8,
                                    int64_t ldk, const float* bw0, const float* bias, int64_t Q, int64_t R, float scale_inv, void* y,
                                    int64_t ldy, int activation, int64_t scaled_cols, float factor, const void* add, int64_t ld_add,
                                    int engine, bsi_stream_t stream) {
    using namespace bsi;
    if ((engine & ~BSI_KEYS_COMPLETE) != BSI_ENGINE_AUTO) return fail(BSI_ERR_INVALID, "linear_rows: engine must be AUTO");
    if (Q < 0 || R < 0 || D <= 0 || ldx < D) return fail(BSI_ERR_INVALID, "linear_rows: bad sizes");
    if (Q == 0 || R == 0) return BSI_OK;
    if (x == nullptr || k8 == nullptr || bw0 == nullptr || y == nullptr) return fail(BSI_ERR_INVALID, "linear_rows: null pointer");
    const int64_t chunks = (D + 255) / 256;
    if (ldk < chunks * 256 || (ldk & 15) || (reinterpret_cast<uintptr_t>(k8) & 15))
        return fail(BSI_ERR_INVALID, "linear_rows: k8 needs 16-byte aligned rows of at least 256*chunks bytes");
    if (ldy < R) return fail(BSI_ERR_INVALID, "linear_rows: ldy < R");
    if (bits < 2 || bits > 8) return fail(BSI_ERR_UNSUPPORTED, "linear_rows: bits must be in [2, 8]");
    if (decimal_places < 0 || decimal_places > 8) return fail(BSI_ERR_UNSUPPORTED, "linear_rows: decimal_places must be in [0, 8]");
    if (activation != BSI_ACT_NONE && activation != BSI_ACT_RELU) return fail(BSI_ERR_INVALID, "linear_rows: unknown activation");
    if (scaled_cols < 0 || scaled_cols > R) return fail(BSI_ERR_INVALID, "linear_rows: bad scaled_cols");
    if (x_dtype != BSI_DTYPE_F32 && x_dtype != BSI_DTYPE_F16 && x_dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_INVALID, "linear_rows: unknown x_dtype");
    if (add != nullptr && ld_add < R) return fail(BSI_ERR_INVALID, "linear_rows: ld_add < R");
    RowsPlan plan;
    if (Q > (1 << 16) || R >= (1 << 24) || chunks >= (1 << 12) || !plan_rows(Q, R, chunks, true, &plan))
        return fail(BSI_ERR_UNSUPPORTED, "linear_rows: not a size for this form");
    if (int rc = require_sm100()) return rc;
    rows::Args a = {};
    a.x = x; a.ldx = ldx; a.D = D; a.bits = bits; a.bw0 = bw0; a.bias = bias;
    a.keys_complete = (engine & BSI_KEYS_COMPLETE) != 0 ? 1 : 0;
    a.Q = static_cast<int>(Q); a.R = static_cast<int>(R); a.chunks = static_cast<int>(chunks);
    a.scale_inv = scale_inv; a.out = y; a.ldo = ldy;
    a.fin = Finishing{activation == BSI_ACT_RELU ? 1 : 0, static_cast<int>(scaled_cols), factor, add, ld_add};
    a.dec_mult = 1;
    for (int i = 0; i < decimal_places; ++i) a.dec_mult *= 10u;
    a.dec_scale = static_cast<double>(a.dec_mult);
    return run_rows(plan, a, nullptr, 0, k8, ldk, x_dtype, x_dtype, static_cast<cudaStream_t>(stream));
}

extern "C" int bsi_b200_debug_last_rows(int* launches_out, int* queries_out, int* parts_out, int* chunks_out, int* stages_out) {
    using namespace bsi;
    if (launches_out == nullptr || queries_out == nullptr || parts_out == nullptr || chunks_out == nullptr || stages_out == nullptr)
        return fail(BSI_ERR_INVALID, "debug_last_rows: null pointer");
    *launches_out = t_rows_launches;
    *queries_out = t_last_rows.nq;
    *parts_out = t_last_rows.parts;
    *chunks_out = t_last_rows.per_part;
    *stages_out = t_last_rows.stages;
    t_rows_launches = 0;
    return BSI_OK;
}

extern "C" int bsi_b200_debug_last_tiles(int* width_out, int* parts_out) {
    using namespace bsi;
    if (width_out == nullptr || parts_out == nullptr) return fail(BSI_ERR_INVALID, "debug_last_tiles: null pointer");
    *width_out = t_last_width;
    *parts_out = t_last_parts;
    return BSI_OK;
}

extern "C" int bsi_b200_debug_exact_int_tiles(unsigned long long* count_out) {
    using namespace bsi;
    if (count_out == nullptr) return fail(BSI_ERR_INVALID, "debug_exact_int_tiles: null pointer");
    BSI_CUDA_TRY(cudaDeviceSynchronize());
    unsigned long long v = 0;
    BSI_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_exact_int_tiles, sizeof(v)));
    const unsigned long long zero = 0;
    BSI_CUDA_TRY(cudaMemcpyToSymbol(g_exact_int_tiles, &zero, sizeof(zero)));
    *count_out = v;
    return BSI_OK;
}
