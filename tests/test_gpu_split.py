"""Dots split along K over a cluster of CTA pairs: same bits as the float32 chain of the CUDA-core engine, with the bounds
holding everywhere and with one row that breaks them (the cluster then falls back to one pair)."""
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


# (columns, parts) of every split kernel and of the unsplit ones next to them; chunk counts that do not divide, a part
# without chunks, ragged rows and columns, shares of 8 and of 16 columns per warp
PLANS = {(512, 2048, 8192): (128, 2), (300, 1111, 5000): (128, 2), (300, 3000, 16384): (256, 2), (256, 1500, 2304): (64, 2),
         (40, 500, 8192): (64, 4), (33, 65, 16384): (64, 4), (300, 500, 16384): (128, 4), (300, 1111, 16384): (256, 4),
         (512, 2040, 4352): (64, 1), (129, 64, 1280): (64, 1), (512, 4000, 1280): (128, 1)}


# broken: the row that breaks every bound, which sends its tiles to one pair and the float32 chain
@pytest.mark.parametrize("broken", [None, 0.5, 1.0])
@pytest.mark.parametrize("Q,R,D", PLANS)
def test_split_dot_and_layer(Q, R, D, broken):
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    width, parts = PLANS[Q, R, D]
    tiles_m, tiles_n = (Q + 255) // 256, (R + width - 1) // width
    exact = tiles_m * tiles_n * 16 * parts                       # warps that add integers: 16 per tile and part
    if broken is not None:
        row = min(int(Q * broken), Q - 1)
        q[row] *= 3.0e4
        exact -= tiles_n * (16 * parts - 14)                     # of the row's tiles the other 14 warps of one pair
    chunks, ld = (D + 255) // 256, (D + 255) // 256 * 256
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    x = q.to(DEV)
    q8 = torch.empty(Q, ld, dtype=torch.int8, device=DEV)
    scales, norms = torch.empty(Q, chunks, device=DEV), torch.empty(Q, chunks, device=DEV)
    bounds = torch.empty(3, R, device=DEV)
    L = capi.lib()
    capi.check(L.bsi_b200_quantize_pack_all(capi.ptr(x), capi.DTYPE_F32, Q, D, D, 2, 7, 1, C.c_float(0.0), None, capi.ptr(scales), None,
                                            capi.ptr(q8), ld, capi.ptr(norms), None, None, capi.stream_ptr()))
    capi.check(L.bsi_b200_key_bounds(capi.ptr(kb["q8"]), ld, R, chunks, capi.ptr(bounds), capi.stream_ptr()))
    want = H.dot_i8(q8, scales, kb["q8"], kb["scales"], o.scale_inv(2), capi.ENGINE_SIMT)
    given = _Bounds(bounds.data_ptr(), norms.data_ptr(), chunks, 64)
    def check_plan():
        assert capi.last_tiles() == (width, parts) and capi.exact_int_tiles() == exact
    capi.exact_int_tiles()
    out = torch.full((Q, R), float("nan"), device=DEV)
    inv = C.c_float(float(o.scale_inv(2)))
    capi.check(L.bsi_b200_dot_i8_bounded(capi.ptr(q8), ld, capi.ptr(scales), chunks, capi.ptr(kb["q8"]), ld, capi.ptr(kb["scales"]), Q, R,
                                         chunks, inv, capi.ptr(out), R, None, 0, C.byref(given), capi.stream_ptr()))
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    check_plan()
    bias = torch.linspace(-1, 1, R, device=DEV)
    for dtype in (torch.float16, torch.bfloat16):
        y = torch.full((Q, R), float("nan"), dtype=dtype, device=DEV)
        capi.check(L.bsi_b200_linear_i8_bounded(capi.ptr(q8), ld, capi.ptr(scales), chunks, capi.ptr(kb["q8"]), ld, capi.ptr(kb["scales"]),
                                                capi.ptr(bias), Q, R, chunks, inv, capi.ptr(y), R, H._DT[dtype], 1, R // 16 * 8, C.c_float(0.3),
                                                C.byref(given),
                                                capi.stream_ptr()))
        z = torch.relu(want.to(dtype) + bias.to(dtype))
        z[:, : R // 16 * 8] *= 0.3
        assert torch.equal(y, z)
        check_plan()
    assert capi.device_status() == 0
