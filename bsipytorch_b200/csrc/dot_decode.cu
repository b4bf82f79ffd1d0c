// Dot of a few query rows (decode batches) with a key set: a stream over the int8 key image.
//
// With 16 or fewer query rows the work is the one read of the keys, R x D bytes; the tensor-core tiles of 256 query rows
// would leave their operand ring 90 % empty rows and, at R = 4096, half of the SMs idle. What bounds this kernel is
// HBM (or L2 for small key sets), so it is organised around bytes in flight:
//
//   * one persistent CTA per SM, 16 warps; a warp's unit of work is one 256-deep chunk of 16 key rows, 4 KB, loaded
//     straight into registers in the A-fragment order of mma.m16n8k32 (keys are the 16 rows, queries the 8 columns);
//     two units per warp are in flight, 128 KB per SM. 16 bytes of one row per lane are two k-steps: the order of k
//     inside a 64-byte span is permuted alike in both operands, which leaves every sum of products unchanged.
//   * K is split over the warps of a CTA (`kw` of them share a row tile), so that 16 rows are enough work for 16 warps.
//     The per-chunk integers meet in shared memory and one thread per output runs the reference's chain over the chunks
//     in order, acc = fmaf(float(I_c), qs[q][c], acc) (bsi_cuda_kernels_dot.cuh:1519-1526): same bits as every engine.
//   * the queries live in shared memory for a slab of K at a time; with more than one slab the running sums of the
//     CTA's outputs are kept in shared memory between slabs.
//   * the layer forms take the activations themselves where quantising them in every CTA is cheap (kFuse): one launch
//     instead of two, and the key loads run under the quantisation.
//
// The legacy int8 MMA of this chip costs about 64 cycles per m16n8k32 and SM quarter: hidden behind HBM up to 8 rows, the
// bound from 16 on (4096 x 16384: 15.1 us at 1 row, 20.4 at 16, 35 at 32), which is where this kernel ends.
#include "common.cuh"
#include "epilogue.cuh"
#include "quantise.cuh"

namespace bsi {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kPitch = 20;              // ints between the 16-key columns of two queries: conflict-free fragment stores
constexpr int kSmemLimit = 232448;
constexpr int kMaxQueries = 16;

struct DecodeArgs {
    const int8_t* a8;          // packed queries (not kFuse)
    int64_t lda;
    const void* x;             // activations (kFuse)
    int64_t ldx, D;
    double dec_scale;
    uint32_t dec_mult;
    int bits;
    const float* qs;           // not kFuse
    int64_t qs_stride;
    const int8_t* k8;
    int64_t ldk;
    int keys_complete;         // nothing on the stream may still be writing k8
    const float* bw0;
    const float* bias;
    int Q, R, chunks;
    int slab, slabs;           // chunks per slab, slabs
    int kw_log2, rt;           // warps along K, row tiles of a CTA's group
    int tiles, groups;         // row tiles, groups of rt tiles
    float scale_inv;
    void* out;
    int64_t ldo;
    Finishing fin;
};

__device__ __forceinline__ uint4 ld_stream(const int8_t* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16-byte piece `u` (0..15) of a query's chunk: odd rows swap 64-byte halves so that the eight lanes of a
// shared-memory phase, two rows of 64 bytes, hit different banks.
__device__ __forceinline__ int query_piece(int row, int u) { return u ^ ((row & 1) << 2); }

// NT: groups of 8 query rows. XT: activation type of the fused form, void otherwise.
// ADD: a matrix is added to the finished values. An instantiation of its own: as a branch in the last loop it cost the dots of 9 to
// 16 rows without one 4 % of 36 MB of keys (9000 x 4096, 16 rows: 11.1 -> 11.6 us) and 20 % of large sets (44000 x 4096: 37.5
// -> 46.2).
template <int NT, typename OutT, typename XT, bool ADD>
__global__ void __launch_bounds__(kThreads, 1) dot_decode_kernel(const DecodeArgs p) {
    constexpr bool kFuse = !std::is_same<XT, void>::value;
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* qbuf = smem;                                                              // [NT * 8][slab][256]
    float* qsc = reinterpret_cast<float*>(qbuf + NT * 8 * p.slab * 256);              // [NT * 8][slab]
    int* ibuf = reinterpret_cast<int*>(qsc + NT * 8 * p.slab);                        // [2][rt][slab][NT * 8][kPitch]
    const int itile = p.slab * NT * 8 * kPitch;                                       // ints of one row tile
    float* accs = reinterpret_cast<float*>(ibuf + 2 * p.rt * itile);                  // [iterations][rt][Q][16], slabs > 1

    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int kw = 1 << p.kw_log2;
    const int ki = warp & (kw - 1);
    const int rt = warp >> p.kw_log2;
    const int g = lane >> 2, t = lane & 3;
    const int iters = (p.groups - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---- the warp's units: chunks ki, ki + kw, ... of each slab, for each of the CTA's groups in turn ----
    auto slab_len = [&](int s) { return min(p.slab, p.chunks - s * p.slab); };
    auto units_in = [&](int s) { return rt < p.rt ? (slab_len(s) - ki + kw - 1) >> p.kw_log2 : 0; };
    int ps = 0, pi = 0, pj = 0;             // next unit to load
    while (ps < p.slabs && units_in(ps) <= 0) ++ps;
    auto load_next = [&](uint4 (&k)[8]) {
        if (ps >= p.slabs) return;
        const int tile = (static_cast<int>(blockIdx.x) + pi * static_cast<int>(gridDim.x)) * p.rt + rt;
        const int r0 = min(tile * 16 + g, p.R - 1), r1 = min(tile * 16 + g + 8, p.R - 1);   // rows beyond R: never stored
        const int64_t off = static_cast<int64_t>(ps * p.slab + ki + (pj << p.kw_log2)) * 256 + t * 16;
        const int8_t* q0 = p.k8 + r0 * p.ldk + off;
        const int8_t* q1 = p.k8 + r1 * p.ldk + off;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            k[2 * s] = ld_stream(q0 + s * 64);
            k[2 * s + 1] = ld_stream(q1 + s * 64);
        }
        if (++pj >= units_in(ps)) {
            pj = 0;
            if (++pi >= iters) {
                pi = 0;
                ++ps;
                while (ps < p.slabs && units_in(ps) <= 0) ++ps;
            }
        }
    };
    uint4 k0[8], k1[8];
    // Programmatic dependent launch: the kernel before this one on the stream, and one more where that is the activation
    // packer, may still run, and what they wrote is visible behind the wait only. That holds for keys too, when one of
    // them builds the image; a caller that has seen the image complete says so, and the first keys are read up here:
    // 16 x 4096 x 16384 bfloat16 layer 19.4 us, 20.8 with every load behind the wait.
    if (p.keys_complete) {
        load_next(k0);
        load_next(k1);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!p.keys_complete) {
        load_next(k0);
        load_next(k1);
    }

    int par = 0;
    for (int s = 0; s < p.slabs; ++s) {
        const int len = slab_len(s), c0 = s * p.slab;
        // ---- the slab's queries and chunk scales ----
        if (s > 0) __syncthreads();      // every warp is done with the previous slab's queries
        if constexpr (kFuse) {
            // a few groups' loads in flight per warp: the loop is latency, not arithmetic
            constexpr int kAhead = sizeof(XT) == 2 ? 4 : 2;
            const float mult = static_cast<float>(p.dec_mult);
            const int total = p.Q * len;
            for (int u0 = warp; u0 < total; u0 += kWarps * kAhead) {
                RawLane<XT> r[kAhead];
#pragma unroll
                for (int h = 0; h < kAhead; ++h) {
                    const int u = min(u0 + h * kWarps, total - 1);
                    const int q = u / len, c = u - q * len;
                    const int64_t col = static_cast<int64_t>(c0 + c) * 256 + lane * 8;
                    const XT* row = behind_wait(static_cast<const XT*>(p.x)) + q * p.ldx;
                    const int64_t left = p.D - col;
                    if (left >= 8 && ((reinterpret_cast<uintptr_t>(row + col) & 15) == 0)) r[h].load(row + col);
                    else r[h].load_tail(row + (left > 0 ? col : 0), left);
                }
#pragma unroll
                for (int h = 0; h < kAhead; ++h) {
                    const int u = u0 + h * kWarps;
                    if (u < total) {
                        const int q = u / len, c = u - q * len;
                        int shift;
                        u64 packed;
                        if (!fast_quantise<XT>(r[h], mult, p.bits, shift, packed))
                            generic_quantise<XT>(r[h].v[0], r[h].v[RawLane<XT>::kVecs - 1], p.dec_scale, p.dec_mult, p.bits, &shift, &packed);
                        *reinterpret_cast<u64*>(qbuf + (q * p.slab + c) * 256 + query_piece(q, lane >> 1) * 16 + (lane & 1) * 8) = packed;
                        if (lane == 0) qsc[q * p.slab + c] = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);
                    }
                }
            }
        } else {
            constexpr int kAhead = 4;
            const int total = p.Q * len * 16;
            for (int i0 = threadIdx.x; i0 < total; i0 += kThreads * kAhead) {
                uint4 v[kAhead];
#pragma unroll
                for (int h = 0; h < kAhead; ++h) {
                    const int i = min(i0 + h * kThreads, total - 1), qc = i >> 4;
                    const int q = qc / len, c = qc - q * len;
                    v[h] = *reinterpret_cast<const uint4*>(behind_wait(p.a8) + q * p.lda + static_cast<int64_t>(c0 + c) * 256 + (i & 15) * 16);
                }
#pragma unroll
                for (int h = 0; h < kAhead; ++h) {
                    const int i = i0 + h * kThreads, qc = i >> 4;
                    if (i < total) {
                        const int q = qc / len, c = qc - q * len;
                        *reinterpret_cast<uint4*>(qbuf + (q * p.slab + c) * 256 + query_piece(q, i & 15) * 16) = v[h];
                    }
                }
            }
            for (int i = threadIdx.x; i < p.Q * len; i += kThreads) {
                const int q = i / len, c = i - q * len;
                qsc[q * p.slab + c] = behind_wait(p.qs)[p.qs_stride ? q * p.qs_stride + c0 + c : q];
            }
        }
        __syncthreads();

        const int mine = units_in(s);
        for (int it = 0; it < iters; ++it) {
            int* ib = ibuf + (it & 1) * p.rt * itile;
            auto unit = [&](uint4 (&k)[8], int c) {
                int d[NT][4];
#pragma unroll
                for (int n = 0; n < NT; ++n) d[n][0] = d[n][1] = d[n][2] = d[n][3] = 0;
#pragma unroll
                for (int sp = 0; sp < 4; ++sp) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        const int q = n * 8 + g;
                        const uint4 b = *reinterpret_cast<const uint4*>(qbuf + (q * p.slab + c) * 256 + query_piece(q, sp * 4 + t) * 16);
                        mma_s8(d[n], k[2 * sp].x, k[2 * sp + 1].x, k[2 * sp].y, k[2 * sp + 1].y, b.x, b.y);
                        mma_s8(d[n], k[2 * sp].z, k[2 * sp + 1].z, k[2 * sp].w, k[2 * sp + 1].w, b.z, b.w);
                    }
                }
                load_next(k);
                int* dst = ib + rt * itile + c * (NT * 8 * kPitch) + g;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    int* col = dst + (n * 8 + 2 * t) * kPitch;
                    col[0] = d[n][0];
                    col[kPitch] = d[n][1];
                    col[8] = d[n][2];
                    col[kPitch + 8] = d[n][3];
                }
            };
            for (int j = 0; j < mine; ++j) {
                const int c = ki + (j << p.kw_log2);
                if (par == 0) unit(k0, c); else unit(k1, c);
                par ^= 1;
            }
            // One barrier per group: a buffer is written again two groups later, behind the next group's barrier, which
            // every thread reaches only after it has read this one.
            __syncthreads();
            const int group = static_cast<int>(blockIdx.x) + it * static_cast<int>(gridDim.x);
            for (int i = threadIdx.x; i < p.rt * p.Q * 16; i += kThreads) {
                const int key = i & 15, rq = i >> 4;
                const int tile_i = rq / p.Q, q = rq - tile_i * p.Q;
                const int row = (group * p.rt + tile_i) * 16 + key;
                const bool last = s + 1 == p.slabs;
                float w = 0.0f, bv = 0.0f;
                OutT av = static_cast<OutT>(0.0f);
                if (last && row < p.R) {
                    w = behind_wait(p.bw0)[row];
                    if (p.bias != nullptr) bv = behind_wait(p.bias)[row];
                    if (ADD) av = behind_wait(static_cast<const OutT*>(p.fin.add))[q * p.fin.ld_add + row];
                }
                float* keep = accs + (static_cast<int64_t>(it) * p.rt * p.Q + rq) * 16 + key;
                float acc = s > 0 ? *keep : 0.0f;
                const int* src = ib + tile_i * itile + q * kPitch + key;
                const float* sc = qsc + q * p.slab;
#pragma unroll 4
                for (int c = 0; c < len; ++c)
                    acc = __fmaf_rn(static_cast<float>(src[c * (NT * 8 * kPitch)]), sc[c], acc);
                if (!last) *keep = acc;
                else if (row < p.R) {
                    const OutT y = scaled_if<OutT>(relu_if<OutT>(finish<OutT>((acc * w) * p.scale_inv, bv, p.bias != nullptr), p.fin.relu != 0),
                                                   row < p.fin.scaled_cols, p.fin.factor);
                    static_cast<OutT*>(p.out)[q * p.ldo + row] = ADD ? plus<OutT>(y, av) : y;
                }
            }
        }
    }
}

template <int NT, typename OutT, typename XT, bool ADD>
int launch_decode_form(const DecodeArgs& a, unsigned grid, int smem, cudaStream_t stream) {
    static int allowed[64] = {0};
    int dev = 0;
    BSI_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || allowed[dev] == 0) {
        BSI_CUDA_TRY(cudaFuncSetAttribute(dot_decode_kernel<NT, OutT, XT, ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
        if (dev >= 0 && dev < 64) allowed[dev] = 1;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    BSI_CUDA_TRY(cudaLaunchKernelEx(&cfg, dot_decode_kernel<NT, OutT, XT, ADD>, a));
    return check_launch("dot_i8 decode launch");
}
template <int NT, typename OutT, typename XT>
int launch_decode(const DecodeArgs& a, unsigned grid, int smem, cudaStream_t stream) {
    return a.fin.add != nullptr ? launch_decode_form<NT, OutT, XT, true>(a, grid, smem, stream)
                                : launch_decode_form<NT, OutT, XT, false>(a, grid, smem, stream);
}

// Splits the work: slabs of K that fit shared memory, warps along K, row tiles per CTA. Returns the shared memory
// in bytes, 0 when the running sums of a many-slab problem do not fit.
int plan_decode(DecodeArgs* a, int nt, unsigned* grid) {
    const int sms = sm_count();
    a->tiles = (a->R + 15) / 16;
    // At most 64 KB of queries at a time: what shared memory does not take is L1, and the key loads in flight need their
    // lines there (16384 x 4096, one row: 25.3 us with 128 KB slabs, 17.7 us with 64 KB, 20.9 us with 32 KB).
    for (int most = 32 / nt; most >= 2; most >>= 1) {
        a->slabs = (a->chunks + most - 1) / most;
        a->slab = (a->chunks + a->slabs - 1) / a->slabs;
        a->kw_log2 = 0;
        while (a->kw_log2 < 4 && (1 << a->kw_log2) < a->slab) ++a->kw_log2;
        const int most_rt = kWarps >> a->kw_log2;
        a->rt = (a->tiles + sms - 1) / sms;                  // no more tiles per CTA than it takes to use every SM
        if (a->rt > most_rt) a->rt = most_rt;
        a->groups = (a->tiles + a->rt - 1) / a->rt;
        *grid = static_cast<unsigned>(a->groups < sms ? a->groups : sms);
        const int64_t iters = (a->groups + *grid - 1) / *grid;
        const int64_t bytes = static_cast<int64_t>(nt) * 8 * a->slab * (256 + 4) +
                              2ll * a->rt * a->slab * nt * 8 * kPitch * 4 +
                              (a->slabs > 1 ? iters * a->rt * a->Q * 16 * 4 : 0);
        if (bytes <= kSmemLimit) return static_cast<int>(bytes);
    }
    return 0;
}

}  // namespace

// Whether a dot of these sizes goes to the decode kernel (see above for the line at 16 rows).
bool decode_fits(int64_t Q, int64_t R, int64_t chunks) {
    return Q <= kMaxQueries && R <= (1 << 27) && chunks <= 4096;
}

// The share of the kernel's warps that have a chunk of their own: as many warps as the next power of two share a row tile
// (5 chunks: 5 of 8, 9 chunks: 9 of 16).
double decode_share(int64_t Q, int64_t chunks) {
    const int64_t most = Q <= 8 ? 32 : 16, slabs = (chunks + most - 1) / most, slab = (chunks + slabs - 1) / slabs;
    int64_t kw = 1;
    while (kw < kWarps && kw < slab) kw *= 2;
    return static_cast<double>(slab) / static_cast<double>(kw * ((slab + kw - 1) / kw));
}

int dot_decode(const int8_t* a8, int64_t lda, const float* qs, int64_t qs_stride, const int8_t* k8, int64_t ldk, const float* bw0,
               const float* bias, int64_t Q, int64_t R, int64_t chunks, float scale_inv, void* out, int64_t ldo, int y_dtype,
               const Finishing& fin, bool keys_complete, cudaStream_t stream, bool* taken) {
    DecodeArgs a = {};
    a.keys_complete = keys_complete ? 1 : 0;
    a.a8 = a8; a.lda = lda; a.qs = qs; a.qs_stride = qs_stride; a.k8 = k8; a.ldk = ldk; a.bw0 = bw0; a.bias = bias;
    a.Q = static_cast<int>(Q); a.R = static_cast<int>(R); a.chunks = static_cast<int>(chunks);
    a.scale_inv = scale_inv; a.out = out; a.ldo = ldo; a.fin = fin;
    const int nt = Q <= 8 ? 1 : 2;
    unsigned grid = 0;
    const int smem = plan_decode(&a, nt, &grid);
    *taken = smem > 0;
    if (smem == 0) return BSI_OK;
#define BSI_DECODE(NT)                                                                                     \
    (y_dtype == BSI_DTYPE_F32   ? launch_decode<NT, float, void>(a, grid, smem, stream)                    \
     : y_dtype == BSI_DTYPE_F16 ? launch_decode<NT, __half, void>(a, grid, smem, stream)                   \
                                : launch_decode<NT, __nv_bfloat16, void>(a, grid, smem, stream))
    if (nt == 1) return BSI_DECODE(1);
    return BSI_DECODE(2);
#undef BSI_DECODE
}

}  // namespace bsi

extern "C" int bsi_b200_linear_decode(const void* x, int x_dtype, int64_t ldx, int64_t D, int decimal_places, int bits,
                                      const int8_t* k8, int64_t ldk, const float* bw0, const float* bias, int64_t Q, int64_t R,
                                      float scale_inv, void* y, int64_t ldy, int activation, int64_t scaled_cols, float factor,
                                      bsi_stream_t stream) {
    return bsi_b200_linear_decode_engine(x, x_dtype, ldx, D, decimal_places, bits, k8, ldk, bw0, bias, Q, R, scale_inv, y, ldy,
                                         activation, scaled_cols, factor, BSI_ENGINE_AUTO, stream);
}

extern "C" int bsi_b200_linear_decode_engine(const void* x, int x_dtype, int64_t ldx, int64_t D, int decimal_places, int bits,
                                             const int8_t* k8, int64_t ldk, const float* bw0, const float* bias, int64_t Q,
                                             int64_t R, float scale_inv, void* y, int64_t ldy, int activation,
                                             int64_t scaled_cols, float factor, int engine, bsi_stream_t stream) {
    return bsi_b200_linear_decode_add(x, x_dtype, ldx, D, decimal_places, bits, k8, ldk, bw0, bias, Q, R, scale_inv, y, ldy,
                                      activation, scaled_cols, factor, nullptr, 0, engine, stream);
}

extern "C" int bsi_b200_linear_decode_add(const void* x, int x_dtype, int64_t ldx, int64_t D, int decimal_places, int bits,
                                          const int8_t* k8, int64_t ldk, const float* bw0, const float* bias, int64_t Q, int64_t R,
                                          float scale_inv, void* y, int64_t ldy, int activation, int64_t scaled_cols, float factor,
                                          const void* add, int64_t ld_add, int engine, bsi_stream_t stream_) {
    using namespace bsi;
    if ((engine & ~BSI_KEYS_COMPLETE) != BSI_ENGINE_AUTO) return fail(BSI_ERR_INVALID, "linear_decode: engine must be AUTO");
    if (Q < 0 || R < 0 || D <= 0 || ldx < D) return fail(BSI_ERR_INVALID, "linear_decode: bad sizes");
    if (Q == 0 || R == 0) return BSI_OK;
    if (x == nullptr || k8 == nullptr || bw0 == nullptr || y == nullptr) return fail(BSI_ERR_INVALID, "linear_decode: null pointer");
    const int64_t chunks = (D + 255) / 256;
    if (ldk < chunks * 256 || (ldk & 15) || (reinterpret_cast<uintptr_t>(k8) & 15))
        return fail(BSI_ERR_INVALID, "linear_decode: k8 needs 16-byte aligned rows of at least 256*chunks bytes");
    if (ldy < R) return fail(BSI_ERR_INVALID, "linear_decode: ldy < R");
    if (bits < 2 || bits > 8) return fail(BSI_ERR_UNSUPPORTED, "linear_decode: bits must be in [2, 8]");
    if (decimal_places < 0 || decimal_places > 8) return fail(BSI_ERR_UNSUPPORTED, "linear_decode: decimal_places must be in [0, 8]");
    if (activation != BSI_ACT_NONE && activation != BSI_ACT_RELU) return fail(BSI_ERR_INVALID, "linear_decode: unknown activation");
    if (scaled_cols < 0 || scaled_cols > R) return fail(BSI_ERR_INVALID, "linear_decode: bad scaled_cols");
    if (x_dtype != BSI_DTYPE_F32 && x_dtype != BSI_DTYPE_F16 && x_dtype != BSI_DTYPE_BF16)
        return fail(BSI_ERR_INVALID, "linear_decode: unknown x_dtype");
    if (add != nullptr && ld_add < R) return fail(BSI_ERR_INVALID, "linear_decode: ld_add < R");
    if (!bsi_b200_linear_decode_fits(Q, R, D)) return fail(BSI_ERR_UNSUPPORTED, "linear_decode: too many query chunks for this form");
    if (int rc = require_sm100()) return rc;
    DecodeArgs a = {};
    a.keys_complete = (engine & BSI_KEYS_COMPLETE) != 0 ? 1 : 0;
    a.x = x; a.ldx = ldx; a.D = D; a.bits = bits; a.k8 = k8; a.ldk = ldk; a.bw0 = bw0; a.bias = bias;
    a.Q = static_cast<int>(Q); a.R = static_cast<int>(R); a.chunks = static_cast<int>(chunks);
    a.scale_inv = scale_inv; a.out = y; a.ldo = ldy;
    a.fin = Finishing{activation == BSI_ACT_RELU ? 1 : 0, static_cast<int>(scaled_cols), factor, add, ld_add};
    a.dec_mult = 1;
    for (int i = 0; i < decimal_places; ++i) a.dec_mult *= 10u;
    a.dec_scale = static_cast<double>(a.dec_mult);
    unsigned grid = 0;
    const int nt = Q <= 8 ? 1 : 2;
    const int smem = plan_decode(&a, nt, &grid);
    if (smem == 0) return fail(BSI_ERR_UNSUPPORTED, "linear_decode: running sums do not fit shared memory");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
#define BSI_DECODE_FUSED(NT)                                                                                         \
    (x_dtype == BSI_DTYPE_F32   ? launch_decode<NT, float, float>(a, grid, smem, stream)                             \
     : x_dtype == BSI_DTYPE_F16 ? launch_decode<NT, __half, __half>(a, grid, smem, stream)                           \
                                : launch_decode<NT, __nv_bfloat16, __nv_bfloat16>(a, grid, smem, stream))
    return nt == 1 ? BSI_DECODE_FUSED(1) : BSI_DECODE_FUSED(2);
#undef BSI_DECODE_FUSED
}

// Every CTA quantises all Q x chunks groups (16 warps; 128 groups add 3.4 us to 4096 x 4096), which a packing kernel does
// once, in about 1 us beside the dot's set-up. Small key sets take the one launch up to 128 groups all the same: there
// the host's second launch (3 us) is the longer part; sets of 32 MB and more, which keep the GPU busy for longer than the
// host needs, up to 32 groups (8 rows of 4096 x 16384: 19.0 us in one launch, 16.5 us in two).
extern "C" int bsi_b200_linear_decode_fits(int64_t Q, int64_t R, int64_t D) {
    const int64_t chunks = (D + 255) / 256;
    const int64_t most = R * chunks * 256 >= (32 << 20) ? 32 : BSI_B200_DECODE_FUSED_GROUPS;
    return Q >= 1 && Q <= 16 && R <= (1 << 27) && Q * chunks <= most ? 1 : 0;
}
