"""Row-mode packing in one pass: slices, scales, int8 image, slice weights and exactness bounds, against the checker."""
import numpy as np
import pytest
import torch

import _capi_helpers as H
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu


# edges of the kernel's splits: one warp per row up to 4 chunks, then 2, 4 and 8, 8 chunks per warp from 33 chunks on, and
# the two-pass kernel from 16385 elements; ragged tails of a lane, a word and a chunk
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(9, 1), (5, 255), (17, 256), (6, 257), (3, 1023), (3, 2048), (2, 2049), (2, 4103), (2, 8200),
                                    (2, 16384), (2, 16385)])
def test_row_pack_leaves_slices_weights_and_bounds(dtype, rows, D):
    import ctypes as C
    g = torch.Generator().manual_seed(rows * 7 + D)
    x = torch.randn(rows, D, generator=g) * 0.02
    x[0] = 0.0
    x[1, D // 2] = 3.0e5 if dtype != torch.float16 else 6.0e4      # float32: still the 32-bit path; a wide shift
    if rows > 2:
        x[2, -1] = float("inf")                                    # the row's 64-bit path, next to fast rows
        x[2, 0] = float("nan") if D > 1 else x[2, 0]
    x = x.to(dtype)
    bits, W, chunks = 6, (D + 63) // 64, (D + 255) // 256
    xd = x.cuda()
    words = torch.full((rows, bits, W), -1, dtype=torch.int64, device="cuda")
    scales = torch.full((rows,), -1.0, device="cuda")
    weights = torch.full((rows, bits), -1.0, device="cuda")
    bounds = torch.full((3, rows), -1.0, device="cuda")
    q8 = torch.full((rows, chunks * 256), 99, dtype=torch.int8, device="cuda")
    capi.check(capi.lib().bsi_b200_quantize_pack_all(capi.ptr(xd), H._DT[dtype], rows, D, D, 2, bits, 0, C.c_float(0.0),
                                                     capi.ptr(words), capi.ptr(scales), None, capi.ptr(q8), chunks * 256, None,
                                                     capi.ptr(weights), capi.ptr(bounds), capi.stream_ptr()))
    want = o.quantize_pack(x.float().numpy(), 2, bits, False, 0.0)
    np.testing.assert_array_equal(scales.cpu().numpy(), want["scales"])
    np.testing.assert_array_equal(H.as_u64(words), want["words"])
    k = q8.cpu().numpy().astype(np.int64)
    np.testing.assert_array_equal(k[:, :D], want["qvals"])
    assert not k[:, D:].any()
    base = np.array([2.0 ** i for i in range(bits - 1)] + [-2.0 ** (bits - 1)], dtype=np.float32)
    np.testing.assert_array_equal(weights.cpu().numpy(), base * want["scales"].reshape(-1, 1))
    per_chunk = np.abs(k).reshape(rows, chunks, 256).sum(2)
    want_b = np.stack([per_chunk.sum(1), per_chunk.max(1), (k * k).sum(1)]).astype(np.float32)
    np.testing.assert_array_equal(bounds.cpu().numpy(), want_b)
    again = torch.empty_like(bounds)
    capi.check(capi.lib().bsi_b200_key_bounds(capi.ptr(q8), chunks * 256, rows, chunks, capi.ptr(again), capi.stream_ptr()))
    assert torch.equal(again, bounds)
