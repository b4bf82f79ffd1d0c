// Dot of few query rows, and layers whose work is less than a second launch. Included by dot_tcgen05.cu (same translation
// unit: it shares the PTX wrappers and the device status word).
//
// The paired tiles put 256 query rows on the tensor memory's lanes; with few rows most of that is padding, and an activation
// packer goes in front as a launch of its own, which costs the host 3.5 us. Here the operands change places: 128 KEY rows are
// the lanes (A operand, streamed by TMA through a ring), a tile of NQ query rows (16 or 32) the columns. What bounds it is
// the key stream where the key set is large (6.2 TB/s beside a fixed 4 us), launch and latency where it is small.
//
//   warp 0      TMA producer: chunks of 128 key rows x 256 bytes into the ring (kFuse = false: the queries' chunk too)
//   warp 1      TMEM allocation; MMA issuer: per chunk 8 x tcgen05.mma.kind::i8 (M = 128, N = NQ, K = 32)
//   warps 2-5   epilogue, a key row per thread: acc = fmaf(float(I), qs[q][c], acc) for NQ columns, chunk after chunk in
//               order (the reference's order, bsi_cuda_kernels_dot.cuh:1519-1526), then cast, bias and store; for one query
//               a warp writes 32 consecutive outputs
//   warps 6-21  kFuse: quantise the activations (quantise.cuh) straight into the swizzled B operand, chunk by chunk, so that
//               the first MMAs run while later chunks are quantised and no packed image exists in global memory. Every CTA
//               quantises what it needs, 0.6 us per chunk of 16 rows (205 instructions per row), which is why the query
//               tiles are narrow: with tiles of 128 rows a 1024 x 1024 layer took 26 us, with 16 rows 5.5 us.
//
// Split along K (`parts` CTAs of a cluster, where the key tiles leave SMs idle): every part keeps its chunks' integer
// accumulators in TMEM until the part before it hands over the running float32 sums (one bulk copy per warp through
// distributed shared memory), folds its own chunks in and hands on; the last part stores. The chain over the chunks is the
// unsplit one, link by link: same bits, no bounds needed.
//
// A CTA has its SM to itself: all of TMEM and so much shared memory that no other kernel that allocates tensor memory fits
// beside it. (A cluster whose CTAs wait for one another must not share tensor memory with a cluster that does the same.) The
// next launch may start (griddepcontrol.launch_dependents) behind the allocation, for the same reason.
// All waits are bounded; a timeout raises the CTA's abort flag and every role drains out, a cluster's other CTAs by their own.
#pragma once

namespace rows {

constexpr int kEpiWarps = 4;
constexpr int kFirstEpi = 2;
constexpr int kQuantWarps = 16;
constexpr int kFirstQuant = 6;
constexpr int kMaxBufs = 16;                              // chunk accumulators in TMEM
constexpr int kMaxStages = 8;                             // chunks in the operand ring
constexpr int kABytes = 2 * 128 * BK;                     // 128 key rows of a chunk: two swizzled k-blocks
constexpr int kSmemBytes = 232448;                        // 227 KB: the most one CTA can opt in to
constexpr int kTmemCols = 512;
constexpr int kBarWords = kMaxStages + 2 * kMaxBufs + kEpiWarps + 1;
constexpr int kFixedBytes = (kBarWords + 1) * 8 + 16;

enum Site { kSiteLoad = 32, kSiteFull = 33, kSiteQueries = 34, kSiteFold = 35, kSiteSums = 36 };

struct Args {
    const void* x;             // kFuse: activations
    int64_t ldx, D;
    double dec_scale;
    uint32_t dec_mult;
    int bits;
    const float* qs;           // otherwise: chunk scales of the packed queries
    int64_t qs_stride;
    const float* bw0;
    const float* bias;
    int keys_complete;         // nothing on the stream may still be writing the keys
    int Q, R, chunks;
    int parts, per_part;       // CTAs along K, chunks of each
    int stages, bufs;          // operand ring, accumulators: as many, or (parts > 1) one for each chunk of a part
    float scale_inv;
    void* out;
    int64_t ldo;
    Finishing fin;
};

__device__ __forceinline__ void tmem_ld_cols16(uint32_t taddr, int32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// Lanes whose 8 elements are not all there or not aligned; out of line, so that the common loop stays short.
template <typename XT>
__device__ __noinline__ RawLane<XT> load_ragged(const XT* src, int left) {
    RawLane<XT> r;
    r.load_tail(src, left);
    return r;
}

// A group with NaN, infinity or values beyond the fast path; its shift through `shift`.
template <typename XT>
__device__ __forceinline__ u64 slow_unit(const RawLane<XT>& r, double dec_scale, uint32_t dec_mult, int bits, int& shift) {
    int s;
    u64 packed;
    generic_quantise<XT>(r.v[0], r.v[RawLane<XT>::kVecs - 1], dec_scale, dec_mult, bits, &s, &packed);
    shift = s;
    return packed;
}

template <int NQ, typename OutT, typename XT>
__global__ void __launch_bounds__((2 + kEpiWarps + (std::is_same<XT, void>::value ? 0 : kQuantWarps)) * 32, 1)
dot_rows_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_q, const Args p) {
    constexpr bool kFuse = !std::is_same<XT, void>::value;
    constexpr int kBHalf = NQ * BK;                                   // queries' k-block
    constexpr int kStageBytes = kABytes + 2 * kBHalf;
    constexpr int kSumBytes = NQ * 128;                               // running sums of a warp's 32 key rows

    extern __shared__ __align__(1024) uint8_t smem[];                 // [stages][2 x 128 key rows, 2 x NQ queries][128]
    uint8_t* sums = smem + p.stages * kStageBytes;                    // parts > 1: [kEpiWarps][NQ / 4][32][4] floats
    float* qsc = reinterpret_cast<float*>(sums + (p.parts > 1 ? kEpiWarps * kSumBytes : 0));   // [per_part][NQ]
    uint64_t* bars = reinterpret_cast<uint64_t*>(qsc + p.per_part * NQ);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBarWords);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const uint32_t ring = smem_u32(smem), bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto tfull_bar = [&](int b) { return bar0 + 8u * (kMaxStages + b); };
    auto tempty_bar = [&](int b) { return bar0 + 8u * (kMaxStages + kMaxBufs + b); };
    auto sum_bar = [&](int w) { return bar0 + 8u * (kMaxStages + 2 * kMaxBufs + w); };
    const uint32_t drain_bar = bar0 + 8u * (kBarWords - 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int part = p.parts > 1 ? static_cast<int>(blockIdx.x) % p.parts : 0;      // = rank in the cluster
    const int r0 = static_cast<int>(blockIdx.x) / p.parts * 128;
    const int q0 = static_cast<int>(blockIdx.y) * NQ;
    const int nq = min(NQ, p.Q - q0);                                 // query rows of this tile
    const int c_lo = part * p.per_part;
    const int n_chunks = min(p.per_part, p.chunks - c_lo);            // at least 1
    const int quant = min(kQuantWarps, nq);                           // quantising warps with a row

    if (warp == 0) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
            if (!kFuse) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
            *abort_flag = 0;
        }
        for (int i = lane; i < kBarWords; i += 32) {
            int count = 1;
            if (i < kMaxStages) count = kFuse ? 1 + quant : 1;                           // the producer, and the quantising warps
            else if (i < kMaxStages + kMaxBufs) count = 2;                               // the MMAs, and the issuer (for the scales it saw)
            else if (i < kMaxStages + 2 * kMaxBufs) count = kEpiWarps;
            mbar_init(bar0 + 8u * i, count);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(static_cast<uint32_t>(kTmemCols)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (p.parts > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    auto cluster_ready = [&] {       // every warp once: the other CTAs' barriers are initialised
        __syncwarp();
        if (p.parts > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    };

    // Chunk c may go into its stage: the chunk before it there has been used. With as many accumulators as stages that is
    // when its accumulator is folded, which spares the MMA issuer a wait of its own; the parts of a split cannot wait for
    // that, their accumulators are folded after the last chunk.
    auto stage_free = [&](int c, int site) {
        if (c < p.stages) return true;
        const int old = c - p.stages;
        return p.parts > 1 ? mbar_wait(tfull_bar(old), 0u, abort_flag, site)
                           : mbar_wait(tempty_bar(old % p.stages), static_cast<uint32_t>(old / p.stages) & 1u, abort_flag, site);
    };

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            bool waited = false;
            auto wait_grid = [&] {
                if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
                waited = true;
            };
            auto keys = [&](int c, int s) {
                mbar_expect_tx(full_bar(s), kABytes + (kFuse ? 0 : 2 * kBHalf));
                tma_load_2d(ring + s * kStageBytes, &map_k, (c_lo + c) * 2 * BK, r0, full_bar(s));
                tma_load_2d(ring + s * kStageBytes + kABytes / 2, &map_k, ((c_lo + c) * 2 + 1) * BK, r0, full_bar(s));
            };
            auto queries = [&](int c, int s) {
                if (kFuse) return;
                tma_load_2d(ring + s * kStageBytes + kABytes, &map_q, (c_lo + c) * 2 * BK, q0, full_bar(s));
                tma_load_2d(ring + s * kStageBytes + kABytes + kBHalf, &map_q, ((c_lo + c) * 2 + 1) * BK, q0, full_bar(s));
            };
            if (!p.keys_complete) wait_grid();
            const int first = min(n_chunks, p.stages);
            for (int c = 0; c < first; ++c) keys(c, c);
            if (!kFuse) {
                wait_grid();
                for (int c = 0; c < first; ++c) queries(c, c);
            }
            int s = 0;
            for (int c = first; c < n_chunks; ++c) {
                if (!stage_free(c, kSiteLoad)) break;
                keys(c, s);
                queries(c, s);
                if (++s == p.stages) s = 0;
            }
        }
        cluster_ready();
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        // One wait and one commit per chunk: with waits for stage, slot and accumulator and k-blocks of their own, a chunk took
        // the issuer 950 cycles, twice what the key stream needs.
        constexpr uint32_t idesc = umma_idesc(NQ);
        int s = 0, b = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int c = 0; c < n_chunks; ++c) {
            if (!mbar_wait(full_bar(s), ph, abort_flag, kSiteFull)) { ok = false; break; }
            // between the quantisers' stores, seen through the barrier, and the MMAs' reads
            if (kFuse) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_after();
            const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(b * NQ);
            const uint64_t adesc = umma_desc(ring + s * kStageBytes), bdesc = umma_desc(ring + s * kStageBytes + kABytes);
            if (pair::elect_one()) {
#pragma unroll
                for (int k = 0; k < 2 * BK / UMMA_K; ++k) {
                    // +32 bytes of K inside the swizzle row = +2 in the 16-byte address field; then the second k-block
                    const uint32_t in = 2u * (k % (BK / UMMA_K)), blk = k / (BK / UMMA_K);
                    umma_i8(tmem_d, adesc + in + blk * (kABytes / 2 / 16), bdesc + in + blk * (kBHalf / 16), idesc, k != 0 ? 1u : 0u);
                }
                mbar_arrive(tfull_bar(b));
                umma_commit(tfull_bar(b));
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; ph ^= 1u; }
            if (++b == p.bufs) b = 0;
        }
        if (!ok && lane == 0) {
            umma_commit(drain_bar);
            const long long t0 = clock64();
            while (!mbar_try(drain_bar, 0) && clock64() - t0 < kWaitCycles / 64) {}
        }
        cluster_ready();
    } else if (warp < kFirstQuant) {
        // ---------------- epilogue ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int ew = warp - kFirstEpi;
        const int quad = warp & 3;                       // TMEM lane quadrant this warp may read
        const int row = r0 + quad * 32 + lane;
        const bool has_bias = p.bias != nullptr;
        float w = 0.0f, bv = 0.0f;
        if (row < p.R) {
            w = behind_wait(p.bw0)[row];
            if (has_bias) bv = behind_wait(p.bias)[row];
        }
        if constexpr (!kFuse) {
            for (int i = threadIdx.x - kFirstEpi * 32; i < n_chunks * NQ; i += kEpiWarps * 32) {
                const int c = i / NQ, q = i % NQ;
                qsc[i] = q < nq ? behind_wait(p.qs)[p.qs_stride ? (q0 + q) * p.qs_stride + c_lo + c : q0 + q] : 0.0f;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        }
        float acc[NQ];
        bool ok = true;
        uint8_t* received = sums + ew * kSumBytes + lane * 16;
        if (part > 0) {
            if (lane == 0) mbar_expect_tx(sum_bar(ew), kSumBytes);
            ok = mbar_wait(sum_bar(ew), 0, abort_flag, kSiteSums);
#pragma unroll
            for (int j = 0; j < NQ; j += 4) {
                const float4 v = ok ? *reinterpret_cast<const float4*>(received + j * 128) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                acc[j] = v.x; acc[j + 1] = v.y; acc[j + 2] = v.z; acc[j + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < NQ; ++j) acc[j] = 0.0f;
        }
        ok = __all_sync(0xffffffffu, ok);
        int b = 0;
        uint32_t bph = 0;
        for (int c = 0; c < n_chunks && ok; ++c) {
            if (!mbar_wait(tfull_bar(b), bph, abort_flag, kSiteFold)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(b * NQ);
            const float* sc = qsc + c * NQ;
#pragma unroll
            for (int j = 0; j < NQ; j += 16) {
                int32_t v[16];
                tmem_ld_cols16(taddr + j, v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 s4 = *reinterpret_cast<const float4*>(sc + j + e);
                    acc[j + e] = __fmaf_rn(pair::int_to_float_exact(v[e]), s4.x, acc[j + e]);
                    acc[j + e + 1] = __fmaf_rn(pair::int_to_float_exact(v[e + 1]), s4.y, acc[j + e + 1]);
                    acc[j + e + 2] = __fmaf_rn(pair::int_to_float_exact(v[e + 2]), s4.z, acc[j + e + 2]);
                    acc[j + e + 3] = __fmaf_rn(pair::int_to_float_exact(v[e + 3]), s4.w, acc[j + e + 3]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(b));
            if (++b == p.bufs) { b = 0; bph ^= 1u; }
        }
        cluster_ready();
        // The ring is free, every MMA that reads it is done: the warp's sums go through it, for a bulk copy to the next part
        // or into the loop below. That loop is rolled on purpose: finished straight from the registers, the columns are
        // kilobytes of instructions that run once, and fetching them took 70 ns per column.
        uint8_t* mine = smem + ew * kSumBytes + lane * 16;
        if (ok) {
#pragma unroll
            for (int j = 0; j < NQ; j += 4) *reinterpret_cast<float4*>(mine + j * 128) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        }
        if (part + 1 < p.parts) {
            if (ok) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(pair::map_to_cta(smem_u32(sums) + ew * kSumBytes, part + 1)), "r"(smem_u32(smem) + ew * kSumBytes), "r"(kSumBytes),
                                 "r"(pair::map_to_cta(sum_bar(ew), part + 1)) : "memory");
                __syncwarp();
            }
        } else if (ok && row < p.R) {
            OutT* o = static_cast<OutT*>(p.out) + static_cast<int64_t>(q0) * p.ldo + row;
            const bool relu = p.fin.relu != 0, scaled = row < p.fin.scaled_cols;
            const OutT* a = p.fin.add == nullptr ? nullptr : behind_wait(static_cast<const OutT*>(p.fin.add)) + q0 * p.fin.ld_add + row;
            OutT add[4], add_next[4];      // of the four queries at hand and of the next four
            auto fetch_add = [&](int j, OutT (&to)[4]) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (a != nullptr && j + e < nq) to[e] = a[(j + e) * p.fin.ld_add];
            };
            fetch_add(0, add);
#pragma unroll 1
            for (int j = 0; j < nq; j += 4) {
                fetch_add(j + 4, add_next);
                const float4 v = *reinterpret_cast<const float4*>(mine + j * 128);
                const float sum[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (j + e < nq) {
                        const OutT y = scaled_if<OutT>(relu_if<OutT>(finish<OutT>((sum[e] * w) * p.scale_inv, bv, has_bias), relu), scaled, p.fin.factor);
                        *o = a != nullptr ? plus<OutT>(y, add[e]) : y;
                    }
                    o += p.ldo;
                    add[e] = add_next[e];
                }
            }
        }
    } else if constexpr (kFuse) {
        // ---------------- quantisers ----------------
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int qw = warp - kFirstQuant;
        if (qw < quant) {
            // This warp's rows are qw, qw + quant, ...; its units are those rows of chunk after chunk. kAhead units are in
            // flight, handed from register set to register set in a rolled loop: unrolled, the body is 20 KB of
            // instructions that each warp fetches for itself, and a unit took 0.7 us.
            constexpr int kAhead = sizeof(XT) == 2 ? 3 : 2;
            const int per_chunk = (nq - qw + quant - 1) / quant;
            const float mult = static_cast<float>(p.dec_mult);
            const XT* x = behind_wait(static_cast<const XT*>(p.x)) + (q0 + qw) * p.ldx + c_lo * 256 + lane * 8;
            const int64_t row_step = quant * p.ldx;
            const int left0 = static_cast<int>(min(p.D - (static_cast<int64_t>(c_lo) * 256 + lane * 8), static_cast<int64_t>(1) << 30));
            const bool vec = (p.D & 7) == 0 && (p.ldx * sizeof(XT) & 15) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
            int load_c = 0, load_i = 0;
            const XT* src = x;
            auto fetch = [&](RawLane<XT>& r) {
                if (load_c < n_chunks) {
                    const int left = left0 - load_c * 256;
                    if (vec && left > 0) r.load(src);
                    else r = load_ragged<XT>(src, left);
                }
                src += row_step;
                if (++load_i == per_chunk) {
                    load_i = 0;
                    ++load_c;
                    src = x + load_c * 256;
                }
            };
            RawLane<XT> buf[kAhead];
#pragma unroll
            for (int j = 0; j < kAhead; ++j) fetch(buf[j]);
            const int piece = (lane & 15) >> 1;
            int s = 0;
            for (int c = 0; c < n_chunks; ++c) {
                if (!__all_sync(0xffffffffu, stage_free(c, kSiteQueries))) break;
                uint8_t* block = smem + s * kStageBytes + kABytes + (lane >> 4) * kBHalf + (lane & 1) * 8;
#pragma unroll 1
                for (int q = qw; q < nq; q += quant) {
                    const RawLane<XT> r = buf[0];
#pragma unroll
                    for (int j = 0; j + 1 < kAhead; ++j) buf[j] = buf[j + 1];
                    fetch(buf[kAhead - 1]);
                    const float amax = RawLane<XT>::abs_value(__reduce_max_sync(0xffffffffu, r.abs_max()));
                    int shift = fast_group_shift(amax, mult, p.bits);
                    u64 packed;
                    if (shift >= 0) packed = r.quantise(mult, shift, p.bits);
                    else packed = slow_unit<XT>(r, p.dec_scale, p.dec_mult, p.bits, shift);
                    // 16-byte piece of the row's 128 bytes, swizzled by the row's place in its group of 8
                    *reinterpret_cast<u64*>(block + q * 128 + ((piece ^ (q & 7)) << 4)) = packed;
                    if (lane == 0) qsc[c * NQ + q] = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(s));
                if (++s == p.stages) s = 0;
            }
        }
        cluster_ready();
    }

    __syncwarp();
    if (threadIdx.x == 0 && *abort_flag) {
        // error path only: copies in flight land before the shared memory goes away
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {}
    }
    tc_fence_before();
    __syncthreads();
    // A copy of this CTA's sums may still be on its way: it has landed when its receiver arrives here, which waited for it on its own
    // barrier. The cluster barrier itself releases nothing, and nothing else is written across.
    if (p.parts > 1) pair::cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem_base), "r"(static_cast<uint32_t>(kTmemCols)) : "memory");
    }
}

}  // namespace rows
