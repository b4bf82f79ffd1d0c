"""Store phase of the paired kernel: blocks of its own for early tiles, blocks in the operand ring for a CTA's last one,
clipped edges, rows that do not start on 16 bytes, a row pitch wider than the matrix."""
import ctypes as C

import pytest
import torch

import _capi_helpers as H
import _inputs
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


# more tiles than CTA pairs at every width (11 x 18 tiles at the widest), ragged rows and columns; R and pitch that
# keep rows on 16 bytes and that do not
@pytest.mark.parametrize("width", [64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("R,pitch", [(4424, 4424), (4424, 4440), (4423, 4423)])
def test_float32_stores(width, R, pitch):
    Q, D = 2650, 512
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=R + width, dtype=torch.float32)
    qa, kb = H.quantize_pack(q.to(DEV), 2, 7, True), H.quantize_pack(k.to(DEV), 2, 6, False)
    want = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), capi.ENGINE_SIMT)
    out = torch.full((Q + 1, pitch), -7.0, device=DEV)
    capi.check(capi.lib().bsi_b200_dot_i8(capi.ptr(qa["q8"]), D, capi.ptr(qa["scales"]), D // 256, capi.ptr(kb["q8"]), D,
                                          capi.ptr(kb["scales"]), Q, R, D // 256, C.c_float(float(o.scale_inv(2))), capi.ptr(out),
                                          pitch, None, 3000 + width, capi.stream_ptr()))
    assert torch.equal(out[:Q, :R], want)
    assert bool((out[Q] == -7.0).all()) and bool((out[:, R:] == -7.0).all())
    assert capi.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("Q,R,pitch,skew", [(2650, 4424, 4424, 0), (2650, 4424, 4440, 1), (300, 776, 777, 0), (200, 4423, 4423, 1)])
def test_layer_stores(dtype, Q, R, pitch, skew):
    D = 768
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=R + Q, dtype=torch.float32)
    qa, kb = H.quantize_pack(q.to(DEV), 2, 7, True), H.quantize_pack(k.to(DEV), 2, 6, False)
    dot = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), capi.ENGINE_SIMT)
    bias = torch.linspace(-1, 1, R + 1, device=DEV)[skew:skew + R]           # skew 1: the bias is not on 16 bytes
    out = torch.full((Q + 1, pitch), -7.0, dtype=dtype, device=DEV)
    code = H._DT[dtype]
    for relu in (0, 1):
        want = dot.to(dtype) + bias.to(dtype)
        want = torch.relu(want) if relu else want
        capi.check(capi.lib().bsi_b200_linear_i8_act(capi.ptr(qa["q8"]), D, capi.ptr(qa["scales"]), D // 256, capi.ptr(kb["q8"]), D,
                                                     capi.ptr(kb["scales"]), capi.ptr(bias), Q, R, D // 256,
                                                     C.c_float(float(o.scale_inv(2))), capi.ptr(out), pitch, code, relu,
                                                     capi.stream_ptr()))
        assert torch.equal(out[:Q, :R], want)
        assert bool((out[Q] == -7.0).all()) and bool((out[:, R:] == -7.0).all())
    assert capi.device_status() == 0
