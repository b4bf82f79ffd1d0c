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


def _sum_kinds(q8, scales, k8, width):
    """Warps of float32 sums, of integer sums below 2^22 and of other integer sums, by the bounds that a warp takes over its 32
    rows and its half of a tile's columns."""
    Q, R, chunks = q8.shape[0], k8.shape[0], scales.shape[1]
    k = k8.double().abs().view(R, chunks, 256).sum(2)
    rows = [scales.double().amax(1), scales.double().sum(1), ((q8.double().view(Q, chunks, 256) ** 2).sum(2) * scales.double() ** 2).sum(1)]
    cols = [k.sum(1), k.amax(1), (k8.double() ** 2).sum(1)]
    blocks, halves = (Q + 255) // 256 * 8, -(-R // width) * 2
    rows = [torch.nn.functional.pad(r, (0, blocks * 32 - Q)).view(blocks, 32).amax(1) for r in rows]             # no rows: no sums
    cols = [torch.cat([c, c[-1:].expand(halves * width // 2 - R)]).view(halves, width // 2).amax(1) for c in cols]
    first = torch.minimum(torch.outer(rows[0], cols[0]), torch.outer(rows[1], cols[1])) * 64
    norm = torch.outer(rows[2], cols[2])
    exact = (first < 2.0 ** 24 * 0.999) | (norm < 2.0 ** 48 * 0.999)
    small = (first < 2.0 ** 22 * 0.999) | (norm < 2.0 ** 44 * 0.999)
    return int((~exact).sum()), int(small.sum()), int((exact & ~small).sum())


# Tiles of every width that the rule takes (float32, else), in one wave; the parts along K where the bounds are there. One chunk (no
# main loop), fewer chunks than accumulators, more; clipped rows and columns, a last block of half a row, shares of 48 columns with
# their load of 16; a row beyond every bound (float32 chain next to integer sums), and where scaled sums between 2^22 and 2^24.
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Q,R,D,scale,widths,parts", [
    (40, 200, 256, 1.0, (64, 64), 1), (257, 72, 512, 1.0, (64, 64), 1), (33, 1000, 2304, 1.0, (64, 64), 2), (33, 1000, 1792, 1.0, (64, 64), 1),
    (300, 4424, 768, 1.0, (128, 128), 1), (129, 9464, 1000, 1.0, (128, 128), 1), (129, 9464, 1000, 8.0, (128, 128), 1),
    (250, 16000, 1280, 1.0, (224, 256), 1), (64, 520, 2048, 6.0, (64, 64), 2), (64, 520, 1536, 6.0, (64, 64), 1),
    (200, 6056, 768, 8.0, (96, 128), 1), (130, 12040, 512, 1.0, (192, 256), 1), (100, 10040, 512, 16.0, (192, 256), 1)])
def test_one_tile_per_pair(dtype, Q, R, D, scale, widths, parts):
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
    width = widths[0 if dtype == torch.float32 else 1]
    floats, small, large = _sum_kinds(q8, scales, kb["q8"], width)
    assert floats > 0 and small > 0 and (large > 0 or scale == 1.0)
    capi.exact_int_tiles()
    for with_bounds in (True, False):
        for b, relu, cols, a in ((None, 0, 0, None), (bias, 0, 0, None), (bias, 1, R // 16 * 8, None), (bias, 0, R // 16 * 8, add), (None, 1, 0, add)):
            y = torch.full((Q + 1, R), -7.0, dtype=dtype, device=DEV)
            capi.check(L.bsi_b200_linear_i8_add(capi.ptr(q8), ld, capi.ptr(scales), chunks, capi.ptr(kb["q8"]), ld, capi.ptr(kb["scales"]),
                                                None if b is None else capi.ptr(b), Q, R, chunks, C.c_float(float(o.scale_inv(2))), capi.ptr(y), R,
                                                H._DT[dtype], relu, cols, C.c_float(0.3), None if a is None else capi.ptr(a), R,
                                                C.byref(given) if with_bounds else None, capi.ENGINE_TCGEN05, capi.stream_ptr()))
            wide = widths[1] if a is not None else 256 if width == 224 and not with_bounds else width      # sums: powers of two
            assert capi.last_tiles() == (wide, parts if with_bounds else 1) and (Q + 255) // 256 * -(-R // wide) <= 74      # one wave of pairs
            ints = capi.exact_int_tiles()
            assert ints == 0 if not with_bounds else ints == small + large or wide != width or parts > 1
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
