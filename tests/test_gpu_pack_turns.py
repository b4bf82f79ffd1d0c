"""The packers that take everything a caller asks for at once: query units in turns of two per warp, key rows in one pass."""
import ctypes as C

import numpy as np
import pytest
import torch

import _capi_helpers as H
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _queries(x, bits, words, shifts):
    rows, D = x.shape
    chunks, W = D // 256, D // 64
    t = {"q8": torch.full((rows, D), 99, dtype=torch.int8, device=DEV), "scales": torch.full((rows, chunks), -1.0, device=DEV),
         "norms": torch.full((rows, chunks), -1.0, device=DEV)}
    if words:
        t["words"] = torch.full((rows, bits, W), -1, dtype=torch.int64, device=DEV)
        t["weights"] = torch.full((rows, bits), -1.0, device=DEV)
    sh = torch.zeros(rows, chunks, dtype=torch.int32, device=DEV) if shifts else None
    p = lambda k: capi.ptr(t[k]) if k in t else None      # noqa: E731
    capi.check(capi.lib().bsi_b200_quantize_pack_all(capi.ptr(x), H._DT[x.dtype], rows, D, D, 2, bits, 1, C.c_float(0.0), p("words"), p("scales"),
                                                     None if sh is None else capi.ptr(sh), p("q8"), D, p("norms"), p("weights"), None,
                                                     capi.stream_ptr()))
    return t


# four turns per warp, two, one; a last warp with fewer, a last turn of one unit, a last block with fewer warps; next to them sizes
# just below the rule. The call that asks for the shifts as well takes the other kernels: the same bits.
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(4737, 2048), (2370, 7936), (4736, 1024), (1300, 2048), (4736, 512), (950, 2304), (700, 4352), (4735, 512), (4737, 1792)])
def test_turns_leave_what_the_other_packers_leave(dtype, rows, D):
    g = torch.Generator(device=DEV).manual_seed(rows + D)
    x = torch.randn(rows, D, generator=g, device=DEV)
    x = torch.where(torch.rand(rows, D, generator=g, device=DEV) < 0.01, x * 20.0, x)
    x[0] = 0.0
    x[1, :256] = -0.0
    x[2, 5] = float("inf")                          # first and second unit of a turn on the 64-bit path, both, the last unit
    x[3, 256 + 7] = float("nan")
    x[4, 3], x[4, 300] = -float("inf"), float("nan")
    x[5, D - 1] = float("inf")
    x[6, :512] = 0.64                               # the clamp: 64 of 6 bits and a sign
    x[rows - 1, D - 256:] = -0.635
    x = x.to(dtype)
    for bits in (7, 4):
        for words in (True, False):
            got, want = _queries(x, bits, words, False), _queries(x, bits, words, True)
            for k in want:
                assert torch.equal(got[k], want[k]), (k, bits, words)


# rows of the 64-bit path by a negative NaN and by -inf, without any positive value, of negative zeros; a last block with fewer rows
@pytest.mark.parametrize("rows,D", [(13, 256), (9, 768), (5, 1500), (3, 2048), (3, 3000), (2, 9000)])
def test_key_rows_by_sign(rows, D):
    g = torch.Generator().manual_seed(rows + D)
    x = -torch.rand(rows, D, generator=g) * 0.05
    x[0, D // 3] = -0.0
    x[1] = -0.0
    if rows > 2:
        x.view(torch.int32)[2, D - 1] = -1          # a negative NaN
    if rows > 3:
        x[3, 0] = -float("inf")
        x[4, D // 2] = 0.31
    bits, W, chunks = 6, (D + 63) // 64, (D + 255) // 256
    xd = x.to(DEV)
    t = {"words": torch.full((rows, bits, W), -1, dtype=torch.int64, device=DEV), "scales": torch.full((rows,), -1.0, device=DEV),
         "weights": torch.full((rows, bits), -1.0, device=DEV), "bounds": torch.full((3, rows), -1.0, device=DEV),
         "q8": torch.full((rows, chunks * 256), 99, dtype=torch.int8, device=DEV)}
    capi.check(capi.lib().bsi_b200_quantize_pack_all(capi.ptr(xd), capi.DTYPE_F32, rows, D, D, 2, bits, 0, C.c_float(0.0), capi.ptr(t["words"]),
                                                     capi.ptr(t["scales"]), None, capi.ptr(t["q8"]), chunks * 256, None, capi.ptr(t["weights"]),
                                                     capi.ptr(t["bounds"]), capi.stream_ptr()))
    want = o.quantize_pack(x.numpy(), 2, bits, False, 0.0)
    np.testing.assert_array_equal(t["scales"].cpu().numpy(), want["scales"])
    np.testing.assert_array_equal(H.as_u64(t["words"]), want["words"])
    k = t["q8"].cpu().numpy().astype(np.int64)
    np.testing.assert_array_equal(k[:, :D], want["qvals"])
    assert not k[:, D:].any()
    per_chunk = np.abs(k).reshape(rows, chunks, 256).sum(2)
    np.testing.assert_array_equal(t["bounds"].cpu().numpy(), np.stack([per_chunk.sum(1), per_chunk.max(1), (k * k).sum(1)]).astype(np.float32))
