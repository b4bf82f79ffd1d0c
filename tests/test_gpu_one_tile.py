"""Paired dots of no more tiles than pairs: the last chunk is folded in by the store phase. Same bits as the float32 chain of the
CUDA-core engine, finished by separate operators."""
import ctypes as C

import pytest
import torch

import _capi_helpers as H
import _inputs
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


class _Bounds(C.Structure):
    _fields_ = [("key_bounds", C.c_void_p), ("query_sq", C.c_void_p), ("query_sq_stride", C.c_int64), ("query_abs_max", C.c_int)]


# one chunk (no main loop), fewer chunks than accumulators, more; tiles of 64, 128 and 256 columns; clipped rows and columns, a last
# block of half a row; a row beyond every bound (float32 chain next to integer sums), sums between 2^22 and 2^24
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Q,R,D,scale", [(40, 200, 256, 1.0), (257, 72, 512, 1.0), (33, 1000, 2304, 1.0), (300, 4424, 768, 1.0), (129, 9464, 1000, 1.0),
                                         (250, 16000, 1280, 1.0), (64, 520, 2048, 6.0)])
def test_one_tile_per_pair(dtype, Q, R, D, scale):
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    q *= scale
    q[Q // 2] *= 3.0e4
    chunks, ld = (D + 255) // 256, (D + 255) // 256 * 256
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    x = q.to(DEV)
    q8 = torch.empty(Q, ld, dtype=torch.int8, device=DEV)
    scales, norms, bounds = torch.empty(Q, chunks, device=DEV), torch.empty(Q, chunks, device=DEV), torch.empty(3, R, device=DEV)
    L = capi.lib()
    capi.check(L.bsi_b200_quantize_pack_all(capi.ptr(x), capi.DTYPE_F32, Q, D, D, 2, 7, 1, C.c_float(0.0), None, capi.ptr(scales), None,
                                            capi.ptr(q8), ld, capi.ptr(norms), None, None, capi.stream_ptr()))
    capi.check(L.bsi_b200_key_bounds(capi.ptr(kb["q8"]), ld, R, chunks, capi.ptr(bounds), capi.stream_ptr()))
    dot = H.dot_i8(q8, scales, kb["q8"], kb["scales"], o.scale_inv(2), capi.ENGINE_SIMT)
    g = torch.Generator(device=DEV).manual_seed(R)
    add = torch.randn(Q, R, generator=g, device=DEV).to(dtype)
    bias = torch.linspace(-1, 1, R, device=DEV)
    given = _Bounds(bounds.data_ptr(), norms.data_ptr(), chunks, 64)
    for with_bounds in (True, False):
        for b, relu, cols, a in ((None, 0, 0, None), (bias, 0, 0, None), (bias, 1, R // 16 * 8, None), (bias, 0, R // 16 * 8, add), (None, 1, 0, add)):
            y = torch.full((Q + 1, R), -7.0, dtype=dtype, device=DEV)
            capi.check(L.bsi_b200_linear_i8_add(capi.ptr(q8), ld, capi.ptr(scales), chunks, capi.ptr(kb["q8"]), ld, capi.ptr(kb["scales"]),
                                                None if b is None else capi.ptr(b), Q, R, chunks, C.c_float(float(o.scale_inv(2))), capi.ptr(y), R,
                                                H._DT[dtype], relu, cols, C.c_float(0.3), None if a is None else capi.ptr(a), R,
                                                C.byref(given) if with_bounds else None, capi.ENGINE_TCGEN05, capi.stream_ptr()))
            want = dot.to(dtype)
            if b is not None:
                want = want + b.to(dtype)
            if relu:
                want = torch.relu(want)
            if cols:
                want[:, :cols] *= 0.3
            if a is not None:
                want = want + a
            assert torch.equal(y[:Q], want), (with_bounds, b is not None, relu, cols, a is not None)
            assert bool((y[Q] == -7.0).all())
    assert capi.device_status() == 0


# queries without their sums of squares: the split's vote would fail, so the dot stays whole
def test_no_split_without_sums_of_squares():
    Q, R, D = 512, 2048, 8192
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=3, dtype=torch.float32)
    qa, kb = H.quantize_pack(q.to(DEV), 2, 7, True), H.quantize_pack(k.to(DEV), 2, 6, False)
    bounds = torch.empty(3, R, device=DEV)
    L = capi.lib()
    capi.check(L.bsi_b200_key_bounds(capi.ptr(kb["q8"]), D, R, D // 256, capi.ptr(bounds), capi.stream_ptr()))
    given = _Bounds(bounds.data_ptr(), None, 0, 64)
    out = torch.empty(Q, R, device=DEV)
    capi.check(L.bsi_b200_dot_i8_bounded(capi.ptr(qa["q8"]), D, capi.ptr(qa["scales"]), D // 256, capi.ptr(kb["q8"]), D, capi.ptr(kb["scales"]), Q, R,
                                         D // 256, C.c_float(float(o.scale_inv(2))), capi.ptr(out), R, None, 0, C.byref(given), capi.stream_ptr()))
    assert capi.last_tiles()[1] == 1
    assert torch.equal(out, H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), capi.ENGINE_SIMT))
