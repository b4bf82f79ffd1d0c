// Last step of an output element, shared by the dot kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

// The steps below follow one another and a product of the caller's (sum x weight x scale). Their float32 additions and products
// are the intrinsics that no compiler contracts: a bias, a factor or a residual sum is rounded as by an operator of its own,
// whatever the code around it is specialised to.
namespace bsi {
namespace {

// Last step of one output element. float: the raw dot value (the microbenchmark entry point).
// half / bfloat16: the layer epilogue of the reference, `scores.to(dtype) + bias.to(dtype)`
// (verify_accuracy_bsi.py:193-195): both terms are narrowed first, added, and narrowed again.
template <typename OutT>
__device__ __forceinline__ OutT finish(float v, float bias, bool has_bias);
template <>
__device__ __forceinline__ float finish<float>(float v, float bias, bool has_bias) {
    return has_bias ? __fadd_rn(v, bias) : v;
}
template <>
__device__ __forceinline__ __half finish<__half>(float v, float bias, bool has_bias) {
    const __half h = __float2half_rn(v);
    return has_bias ? __float2half_rn(__fadd_rn(__half2float(h), __half2float(__float2half_rn(bias)))) : h;
}
template <>
__device__ __forceinline__ __nv_bfloat16 finish<__nv_bfloat16>(float v, float bias, bool has_bias) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    return has_bias ? __float2bfloat16_rn(__fadd_rn(__bfloat162float(h), __bfloat162float(__float2bfloat16_rn(bias)))) : h;
}

// max(v, 0) on the finished output value when the layer's activation is fused (NaN stays NaN).
template <typename OutT>
__device__ __forceinline__ OutT relu_if(OutT v, bool relu) {
    return (relu && static_cast<float>(v) < 0.0f) ? static_cast<OutT>(0.0f) : v;
}

// The finished value times a factor, rounded to the output type again: what a separate elementwise multiplication of the
// layer's output by a scalar computes (OPT's query scaling).
template <typename OutT>
__device__ __forceinline__ OutT scaled_if(OutT v, bool on, float factor) {
    return on ? static_cast<OutT>(__fmul_rn(static_cast<float>(v), factor)) : v;
}

// The finished value plus one of another matrix, rounded to the output type: a separate elementwise addition's result.
template <typename OutT>
__device__ __forceinline__ OutT plus(OutT v, OutT add) {
    return static_cast<OutT>(__fadd_rn(static_cast<float>(v), static_cast<float>(add)));
}

}  // namespace
}  // namespace bsi
