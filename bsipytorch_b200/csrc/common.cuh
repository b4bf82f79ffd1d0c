// Shared helpers of the bsi_b200 library: status codes, error recording, launch checks.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/bsi_b200.h"

namespace bsi {

// Thread-local detail of the last failure; read through bsi_b200_last_error().
void set_error(const char* fmt, ...);

inline int fail(int code, const char* what) {
    set_error("%s", what);
    return code;
}

// Checks the launch that was just enqueued (configuration errors surface here).
inline int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: %s", what, cudaGetErrorString(e));
        return BSI_ERR_CUDA;
    }
    return BSI_OK;
}

#define BSI_CUDA_TRY(expr)                                                        \
    do {                                                                          \
        cudaError_t _e = (expr);                                                  \
        if (_e != cudaSuccess) {                                                  \
            ::bsi::set_error("%s: %s", #expr, cudaGetErrorString(_e));            \
            return BSI_ERR_CUDA;                                                  \
        }                                                                         \
    } while (0)

// Number of SMs of the current device (cached per device).
int sm_count();

// 0 when the current device is sm_100 class, an error code otherwise.
int require_sm100();

// Destinations of a linear whose output rows are dealt out to several matrices (n = 0: plain output).
struct ScatterDst {
    int n;
    int rows_per_dst;                 // multiple of 32
    void* y[BSI_B200_MAX_PEERS];      // row q -> y[q / rows_per_dst], local row q % rows_per_dst
};

// Destinations of a linear that re-quantises its finished output (n = 0: off). The output row block of a
// tile is one 256-column chunk per row, so its chunk scale is known inside the tile.
struct RequantDst {
    int n;                 // destinations (own buffer and peer mappings alike)
    int bits;              // 7 for activations
    float mult;            // 10^decimal_places, at most 1000
    int64_t ld8;           // row pitch of the int8 matrices (bytes)
    int64_t scale_ld;      // floats per row of the scale matrices
    int8_t* q8[BSI_B200_MAX_PEERS];      // already offset to this linear's first output column
    float* scales[BSI_B200_MAX_PEERS];   // already offset to this linear's first output chunk
};

// What happens to a finished output value: ReLU, a factor for the first scaled_cols columns (a multiple of 8), and the
// addition of a matrix of the output's type and shape, rounded once more (a residual sum; null: none).
struct Finishing {
    int relu;
    int scaled_cols;
    float factor;
    const void* add;
    int64_t ld_add;
};

// Bounds registered for a key image (bsi_b200_register_key_bounds): with them a dot can tell, per tile, that every
// prefix of a chunk sum stays below 2^24 in magnitude, where integer accumulation gives the float32 chain's bits.
struct KeyBounds {
    const float* abs_sum;    // [3, rows] device: sum of |k| per key row, largest sum over one chunk, sum of k^2
    int64_t rows;
    float query_abs_max;     // largest magnitude of a query integer in dots against these keys
};
bool lookup_key_bounds(const void* k8, KeyBounds* out);   // false: none registered (or BSI_B200_EXACT_INT=0)
struct QueryBounds {
    const float* sq_norms;   // per (row, chunk): (2^shift)^2 * sum of squares of the chunk's integers
    int64_t stride;          // floats per row
};
bool lookup_query_bounds(const void* a8, QueryBounds* out);
bool exact_int_enabled();     // BSI_B200_EXACT_INT is not 0
// The bounds of one dot: what the caller passes (given != nullptr), else what is registered for the two images.
bsi_dot_bounds resolve_bounds(const bsi_dot_bounds* given, const void* a8, const void* k8, int64_t R);

// True unless BSI_B200_PDL=0: the dot kernels are launched with programmatic stream serialisation (their set-up
// may overlap the tail of a dot kernel right before them on the stream).
bool pdl_enabled();

// Reads and clears the status word of the peer barrier kernels (0 = clean, 64 + p = gave up waiting for rank p).
int take_peer_status(int* v);

// For kernels that start while the kernels in front of them on the stream still run (programmatic dependent launch): the
// pointer, behind griddepcontrol.wait, to something those may have written. Loads through it are ordinary coherent ones
// behind the wait. __ldg, and a const __restrict__ parameter, which the compiler treats alike, are no choice there:
// ld.global.nc is for memory that nobody writes while the kernel is resident, and may be moved over the wait.
template <typename T>
__device__ __forceinline__ const T* behind_wait(const T* p) {
    size_t g = __cvta_generic_to_global(p);
    asm volatile("" : "+l"(g) :: "memory");
    return static_cast<const T*>(__cvta_global_to_generic(g));
}

}  // namespace bsi
