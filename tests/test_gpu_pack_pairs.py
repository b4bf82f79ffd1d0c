"""The packer that takes two units per warp (16-bit types, more units than warps are resident): the bits that the same values
give as float32, which go through the kernel with one unit per warp."""
import ctypes as C

import pytest
import torch

from bsipytorch_b200 import capi

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _pack(x, D, bits, words, q8):
    rows, chunks, W = x.shape[0], (D + 255) // 256, (D + 63) // 64
    out = dict(scales=torch.full((rows, chunks), -1.0, device=DEV), norms=torch.full((rows, chunks), -1.0, device=DEV),
               shifts=torch.full((rows, chunks), -1, dtype=torch.int32, device=DEV))
    if words:
        out.update(words=torch.full((rows, bits, W), -1, dtype=torch.int64, device=DEV), weights=torch.full((rows, bits), -1.0, device=DEV))
    if q8:
        out["q8"] = torch.full((rows, chunks * 256), -1, dtype=torch.int8, device=DEV)
    code = {torch.float32: capi.DTYPE_F32, torch.float16: capi.DTYPE_F16, torch.bfloat16: capi.DTYPE_BF16}[x.dtype]
    p = lambda k: capi.ptr(out[k]) if k in out else None                     # noqa: E731
    capi.check(capi.lib().bsi_b200_quantize_pack_all(capi.ptr(x), code, rows, D, x.stride(0), 2, bits, 1, C.c_float(0.0), p("words"),
                                                     p("scales"), p("shifts"), p("q8"), chunks * 256, p("norms"), p("weights"), None,
                                                     capi.stream_ptr()))
    return out


# an odd number of units, odd and even chunks per row (pairs that lie across two rows), ragged depth, a row pitch beyond the
# depth, both 16-byte halves of a lane behind the end. All resident warps together take 9472 units at a time (148 SMs, 4 blocks
# of 8 warps): the last three shapes go two to six turns, rows and chunks carried on by strides that the chunks do not divide
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,D,pitch", [(4737, 256, 256), (1601, 768, 768), (2500, 512, 520), (1300, 1000, 1000), (1211, 1289, 1296), (901, 1541, 1541),
                                          (9001, 1289, 1296), (7001, 768, 768), (3001, 1700, 1700)])
@pytest.mark.parametrize("bits,words,q8", [(7, True, True), (7, False, True), (5, True, False), (8, True, True)])
def test_pairs_equal_single_units(rows, D, pitch, dtype, bits, words, q8):
    g = torch.Generator().manual_seed(rows + D)
    x = torch.randn(rows, pitch, generator=g) * torch.tensor([0.01, 1.0, 30.0])[torch.randint(0, 3, (rows, 1), generator=g)]
    x[::7, D // 2] = float("inf")                 # units of the 64-bit path in either half of a pair, here and there ...
    x[3::11, 0] = float("nan")
    x[rows // 2: rows // 2 + 40] *= 1.0e6         # ... and whole stretches of them
    if rows > 9000 and bits == 8:
        x *= 1.0e6                                # two units in three: more than a warp's queue holds
    x = x.to(dtype).to(DEV)[:, :D]
    got, want = _pack(x, D, bits, words, q8), _pack(x.float(), D, bits, words, q8)
    if rows > 9000 and bits == 8:
        # a warp whose queue overflows takes all its units on the 64-bit path, which leaves infinity ("no sum") for each; which
        # units share a warp differs between the two kernels
        some = torch.isinf(got["norms"]) | torch.isinf(want["norms"])
        assert 0 < some.sum() < some.numel()
        got["norms"][some] = want["norms"][some] = float("inf")
    for k in want:
        assert torch.equal(got[k].view(torch.uint8), want[k].view(torch.uint8)), k
