"""Residual sums in the linears' epilogues: the bits of the linear followed by an elementwise addition."""
import ctypes as C

import pytest
import torch

import _capi_helpers as H
import _inputs
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


# key-streaming kernel, rows kernel, paired tiles of 64, 128 and 256 columns, unsplit and split, ragged columns, a matrix to
# add whose rows are no multiple of 16 bytes, or start off one
# with a bias and without one: there a product stands in front of the addition, and float32 must not contract the two
@pytest.mark.parametrize("biased", [True, False])
@pytest.mark.parametrize("pad,shift", [(0, 0), (3, 0), (8, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Q,R,D", [(5, 300, 768), (20, 500, 1024), (300, 768, 512), (1024, 768, 768), (130, 77, 512), (257, 3000, 512),
                                   (700, 12288, 256), (40, 500, 8192), (300, 3000, 16384)])
def test_linear_plus_matrix(Q, R, D, dtype, pad, shift, biased):
    L = capi.lib()
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    chunks, ld = (D + 255) // 256, (D + 255) // 256 * 256
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    x = q.to(DEV)
    q8 = torch.empty(Q, ld, dtype=torch.int8, device=DEV)
    scales, norms = torch.empty(Q, chunks, device=DEV), torch.empty(Q, chunks, device=DEV)
    bounds = torch.empty(3, R, device=DEV)
    capi.check(L.bsi_b200_quantize_pack_all(capi.ptr(x), capi.DTYPE_F32, Q, D, D, 2, 7, 1, C.c_float(0.0), None, capi.ptr(scales), None,
                                            capi.ptr(q8), ld, capi.ptr(norms), None, None, capi.stream_ptr()))
    capi.check(L.bsi_b200_key_bounds(capi.ptr(kb["q8"]), ld, R, chunks, capi.ptr(bounds), capi.stream_ptr()))

    class Bounds(C.Structure):
        _fields_ = [("key_bounds", C.c_void_p), ("query_sq", C.c_void_p), ("query_sq_stride", C.c_int64), ("query_abs_max", C.c_int)]

    given = Bounds(bounds.data_ptr(), norms.data_ptr(), chunks, 64)
    bias = torch.linspace(-1, 1, R, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(Q + R)
    flat = torch.randn(Q * (R + pad) + shift, generator=g, device=DEV).to(dtype)
    add = flat[shift:].view(Q, R + pad)[:, :R]

    def linear(matrix, ld_add, relu, factor=0.3):
        y = torch.full((Q, R), float("nan"), dtype=dtype, device=DEV)
        capi.check(L.bsi_b200_linear_i8_add(capi.ptr(q8), ld, capi.ptr(scales), chunks, capi.ptr(kb["q8"]), ld, capi.ptr(kb["scales"]),
                                            capi.ptr(bias) if biased else None, Q, R, chunks, C.c_float(float(o.scale_inv(2))), capi.ptr(y), R,
                                            H._DT[dtype], relu, R // 16 * 8 if factor else 0, C.c_float(factor), matrix, ld_add, C.byref(given), 0, capi.stream_ptr()))
        return y

    for relu, factor in ((0, 0.3), (1, 0.3), (0, 0.0)):
        assert torch.equal(linear(capi.ptr(add), R + pad, relu, factor), linear(None, 0, relu, factor).add_(add))
    assert capi.device_status() == 0


# the one-launch forms
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Q,R,D", [(3, 300, 1024), (16, 130, 2048), (21, 300, 1024), (64, 777, 2816), (512, 1100, 1000)])
def test_one_launch_plus_matrix(Q, R, D, dtype):
    L = capi.lib()
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    x = q.to(dtype).to(DEV)
    call = L.bsi_b200_linear_rows if Q > 16 else L.bsi_b200_linear_decode_add
    add = torch.randn(Q, R, generator=torch.Generator(device=DEV).manual_seed(Q), device=DEV).to(dtype)

    def linear(matrix, factor):
        y = torch.full((Q, R), float("nan"), dtype=dtype, device=DEV)
        capi.check(call(capi.ptr(x), H._DT[dtype], D, D, 2, 7, capi.ptr(kb["q8"]), kb["q8"].shape[1], capi.ptr(kb["scales"]), None, Q, R,
                        C.c_float(float(o.scale_inv(2))), capi.ptr(y), R, 0, 8 if factor else 0, C.c_float(factor), matrix, R, 0, capi.stream_ptr()))
        return y

    for factor in (0.3, 0.0):
        assert torch.equal(linear(capi.ptr(add), factor), linear(None, factor).add_(add))
    assert capi.device_status() == 0
