"""Dots with key bounds but without the queries' sums of squares: split along K only where the cheap bounds may carry the vote. The
bits are those of the CUDA-core engine whether it passes or fails."""
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


# four parts from 24 chunks on, two from 48, and just below; tiles that a split would have to widen; even activations, a row beyond
# every bound among them, outliers all over
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("Q,R,chunks,parts", [(64, 512, 24, 4), (64, 512, 23, 1), (300, 256, 64, 4), (40, 2048, 48, 2), (40, 2048, 47, 1), (512, 2048, 32, 1)])
def test_split_without_sums(dtype, Q, R, chunks, parts):
    D, L = chunks * 256, capi.lib()
    for values in ("even", "one row", "outliers"):
        q, k = (_inputs.fc1 if values == "outliers" else _inputs.fc2)(Q=Q, R=R, D=D, seed=R + chunks, dtype=torch.float32)
        if values == "one row":
            q[Q // 2] *= 3.0e4
        qa, kb = H.quantize_pack(q.to(DEV), 2, 7, True), H.quantize_pack(k.to(DEV), 2, 6, False)
        bounds = torch.empty(3, R, device=DEV)
        capi.check(L.bsi_b200_key_bounds(capi.ptr(kb["q8"]), D, R, chunks, capi.ptr(bounds), capi.stream_ptr()))
        given = _Bounds(bounds.data_ptr(), None, 0, 64)
        y = torch.full((Q, R), -7.0, dtype=dtype, device=DEV)
        capi.exact_int_tiles()
        capi.check(L.bsi_b200_linear_i8_bounded(capi.ptr(qa["q8"]), D, capi.ptr(qa["scales"]), chunks, capi.ptr(kb["q8"]), D, capi.ptr(kb["scales"]), None,
                                                Q, R, chunks, C.c_float(float(o.scale_inv(2))), capi.ptr(y), R, H._DT[dtype], 0, 0, C.c_float(1.0),
                                                C.byref(given), capi.stream_ptr()))
        assert capi.last_tiles()[1] == parts
        ints, tiles = capi.exact_int_tiles(), (Q + 255) // 256 * ((R + 63) // 64)
        if parts > 1 and values == "even":      # the vote passed everywhere: 16 epilogue warps a pair, those without rows too
            assert ints == 16 * parts * tiles
        if parts > 1 and values == "one row":   # and failed in one row of tiles
            assert ints < 16 * parts * tiles
        want = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), capi.ENGINE_SIMT).to(dtype)
        assert torch.equal(y, want)
    assert capi.device_status() == 0
