"""The rows kernel (key rows on the tensor memory's lanes): one-launch layers of more than 16 rows and dots of few rows give
the bits of the paired tensor-core tiles."""
import pytest
import torch

import _capi_helpers as H
import _inputs
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one row beyond a tile of 16, tiles of 32 rows (more than 148 of 16), 128 and 129 keys, one chunk, operand rings that turn
# over (more than 6 chunks), also of parts along K, whose stages are free once multiplied (8 and 7 chunks in a ring of 6), two and
# four parts with a shorter last one, ragged depth, keys and rows; plan: query rows of a tile, parts, chunks of a part, ring
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Q,R,D,plan", [(17, 128, 256, (16, 1, 1, 1)), (33, 129, 250, (16, 1, 1, 1)), (512, 1100, 1000, (32, 1, 4, 4)),
                                        (600, 500, 760, (32, 1, 3, 3)), (77, 777, 1000, (16, 2, 2, 2)), (20, 9000, 2000, (16, 1, 8, 6)),
                                        (16, 2300, 2304, (16, 3, 3, 3)), (64, 700, 2800, (16, 4, 3, 3)), (13, 3000, 3840, (16, 4, 4, 4)),
                                        (40, 130, 4096, (16, 4, 4, 4)), (64, 2048, 4096, (16, 2, 8, 6)), (50, 1999, 3835, (16, 2, 8, 6))])
def test_one_launch_layer_of_many_rows(dtype, Q, R, D, plan, monkeypatch):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    assert capi.lib().bsi_b200_linear_rows_fits(Q, R, D) == 1
    capi.last_rows()
    x, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    x[1] *= 3.0e3 if dtype == torch.float16 else 3.0e4        # sums beyond 2^24: the order of the chunks shows
    x[2, D // 3] = float("inf")
    x[2, 5] = float("nan")
    x = x.to(dtype).to(DEV)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    bias = torch.linspace(-1, 1, R, device=DEV)
    wide = torch.zeros(Q, D + 3, dtype=dtype, device=DEV)
    wide[:, :D] = x                                           # rows that are not 16-byte aligned
    for b in (None, bias):
        monkeypatch.setenv("BSI_B200_ENGINE", "tcgen05")
        want = ops.bsi_layer_forward(x, keys, b, 2)
        monkeypatch.delenv("BSI_B200_ENGINE")
        assert capi.last_rows()[0] == 0
        for _ in range(3):                                    # the later calls read keys ahead of the wait
            assert torch.equal(ops.bsi_layer_forward(x, keys, b, 2), want)
            torch.cuda.synchronize()
        assert torch.equal(ops.bsi_layer_forward(wide[:, :D], keys, b, 2), want)
        assert capi.last_rows() == (4,) + plan
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = [ops.bsi_layer_forward(x, keys, bias, 2) for _ in range(3)]
    graph.replay()
    assert all(torch.equal(y, want) for y in captured)
    assert capi.device_status() == 0


# packed queries: both tile widths, a row that makes every bound fail, parts along K, one scale per row, no room for a split
@pytest.mark.parametrize("chunk_mode", [True, False])
@pytest.mark.parametrize("Q,R,D", [(17, 300, 512), (32, 129, 4096), (20, 2100, 8192), (24, 4111, 4352), (1, 10240, 768), (16, 10300, 4096),
                                   (9, 12288, 4096), (32, 19000, 2560)])
def test_packed_dot_of_few_rows(Q, R, D, chunk_mode):
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    if Q > 1:
        q[1] *= 3.0e4
    qa = H.quantize_pack(q.to(DEV), 2, 7, chunk_mode)
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    capi.last_rows()
    got = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2))
    assert capi.last_rows()[:2] == (1, 16 if Q <= 16 else 32)
    want = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), 3064)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert capi.device_status() == 0


# deep K over few key tiles: the paired tiles split along K add all parts at once, where their bounds are given and read as
# whole vectors; from 16 key tiles on, at fewer chunks or without bounds the rows kernel
@pytest.mark.parametrize("Q,R,D,rows", [(32, 512, 8192, 0), (17, 130, 8192, 0), (32, 960, 16384, 0), (24, 2048, 8192, 1), (32, 512, 4096, 1),
                                        (32, 512, 7936, 1)])
def test_deep_dots_of_few_keys_take_the_shorter_way(Q, R, D, rows):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    queries = ops.build_bsi_queries_cuda_batch_packed(q.to(DEV), 2)
    capi.last_rows()
    got = ops.batch_dot_product_multiquery_cuda_batch_caps(queries, keys)[0]
    assert capi.last_rows()[0] == rows
    if not rows:
        assert capi.last_tiles()[1] > 1
    t, b = ops.debug_query_batch_tensors(queries), ops.debug_keys_tensors(keys)
    call = lambda: H.dot_i8(t["q8"], t["scales"], b["q8"], b["scales"].reshape(-1), o.scale_inv(2))      # noqa: E731
    assert torch.equal(call().view(torch.int32), got.view(torch.int32))
    assert capi.last_rows()[0] == 1                            # no bounds: no split
    assert capi.device_status() == 0


# up to 16 rows and more key tiles than SMs: the key-streaming kernel, but for chunks that leave its warps idle (5 of 8, 10 of 16) and
# for long waves that are nearly full
@pytest.mark.parametrize("Q,R,D,rows", [(1, 18944, 512, 1), (1, 18945, 512, 0), (8, 50272, 768, 0), (16, 19072, 4096, 0), (16, 28416, 4096, 1), (8, 28416, 4096, 0), (16, 20000, 1280, 1),
                                        (3, 37888, 4096, 1), (9, 20001, 2560, 1), (16, 19000, 6912, 1), (4, 19000, 6912, 0)])
def test_few_rows_and_more_key_tiles_than_sms(Q, R, D, rows):
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    qa = H.quantize_pack(q.to(DEV), 2, 7, True)
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    capi.last_rows()
    got = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2))
    assert capi.last_rows()[0] == rows
    want = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), 3064)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert capi.device_status() == 0


# where a CTA's share of the quantisation outweighs a second launch, tiles of 32 rows and five chunks among them, a depth of no
# whole vectors, and where the key-streaming kernel has its own form or packed rows are read faster
def test_one_launch_rule():
    L = capi.lib()
    fits, replayed = L.bsi_b200_linear_rows_fits, lambda *size: L.bsi_b200_linear_rows_ways(*size) >> 1      # noqa: E731
    assert [fits(64, 4096, 4096), fits(64, 2048, 2048), fits(512, 4096, 4096), fits(16, 256, 256), fits(17, 256, 256)] == [0, 1, 0, 0, 1]
    assert [fits(374, 739, 3055), fits(56, 7808, 1280), fits(24, 16256, 1280), fits(48, 7552, 1024)] == [0, 0, 1, 1]
    assert [fits(14, 207, 3291), fits(14, 207, 3328), fits(16, 2185, 4352), fits(9, 8960, 5104), fits(4, 11000, 4096)] == [0, 1, 0, 1, 0]
    h, f = capi.DTYPE_F16, capi.DTYPE_F32
    assert [replayed(512, 1024, 1024, h), replayed(512, 1024, 1024, f), replayed(432, 660, 768, h), replayed(64, 2048, 2048, h),
            replayed(24, 16256, 1280, h), replayed(13, 3000, 3840, h)] == [0, 1, 1, 1, 1, 0]


# the route a captured layer takes: more than 32 rows in tiles of 32 go to packer and paired tiles, the bits are the same
@pytest.mark.parametrize("dtype,Q,R,D,rows", [(torch.float16, 472, 640, 768, 0), (torch.bfloat16, 232, 1920, 256, 0), (torch.float32, 232, 1920, 256, 1),
                                              (torch.float16, 64, 777, 2816, 1)])
def test_captured_layers_take_the_shorter_way(dtype, Q, R, D, rows):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    x, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=dtype)
    x, bias = x.to(DEV), torch.linspace(-1, 1, R, device=DEV)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    capi.last_rows()
    want = ops.bsi_layer_forward(x, keys, bias, 2)
    assert capi.last_rows()[0] == 1
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ops.bsi_layer_forward(x, keys, bias, 2)
    assert capi.last_rows()[0] == rows
    graph.replay()
    assert torch.equal(got, want)
    assert capi.device_status() == 0
