"""The decode kernel (16 query rows and fewer): same bits as the checker and as the tensor-core tiles."""
import numpy as np
import pytest
import torch

import _capi_helpers as H
import _inputs
from bsipytorch_b200 import capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


# edges of the splits: query groups of 8, row tiles of 16, more tiles than SMs (two and more per CTA), warps along K
# (1, 2, 16 chunks and one more), slabs of K (32 chunks at 8 rows, 16 at 16), ragged depth, the first size beyond
@pytest.mark.parametrize("Q,R,D", [(1, 1, 256), (1, 17, 250), (8, 300, 512), (9, 300, 4096), (16, 5000, 768), (17, 4111, 4352),
                                   (16, 500, 8192), (16, 2500, 4352), (3, 40, 16384), (5, 2400, 33000)])
@pytest.mark.parametrize("chunk_mode", [True, False])
def test_decode_dot_matches_other_engines(Q, R, D, chunk_mode):
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    qa = H.quantize_pack(q.to(DEV), 2, 7, chunk_mode)
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    got = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2))
    want = H.dot_i8(qa["q8"], qa["scales"], kb["q8"], kb["scales"], o.scale_inv(2), 3064)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert capi.device_status() == 0


# the one-launch layer: 1 .. 128 (row, chunk) groups per CTA, chunks that need the 64-bit quantiser, ragged depth
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Q,R,D", [(1, 33, 256), (1, 3000, 4096), (2, 520, 16384), (7, 100, 1000), (8, 2500, 4096), (16, 130, 2048),
                                   (2, 8192, 4096), (8, 8191, 4096)])
def test_one_launch_layer_equals_build_and_dot(dtype, Q, R, D):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    assert capi.lib().bsi_b200_linear_decode_fits(Q, R, D) == 1
    q, k = _inputs.fc1(Q=Q, R=R, D=D, seed=Q + R + D, dtype=torch.float32)
    if Q > 1:
        q[1, D // 3] = float("inf")
        q[1, 5] = float("nan")
        q[0, D - 1] = 6.0e4
    x = q.to(dtype).to(DEV)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    bias = torch.linspace(-1, 1, R, device=DEV)
    scores = ops.batch_dot_product_multiquery_cuda_batch_caps(ops.build_bsi_queries_cuda_batch_packed(x, 2), keys)[0]
    for b in (None, bias):
        want = scores.to(dtype) if b is None else scores.to(dtype) + b.to(dtype)
        got = ops.bsi_layer_forward(x, keys, b, 2)
        assert got.dtype == dtype and torch.equal(got, want)
        strided = torch.zeros(Q, D + 3, dtype=dtype, device=DEV)
        strided[:, :D] = x
        assert torch.equal(ops.bsi_layer_forward(strided[:, :D], keys, b, 2), want)     # rows that are not 16-byte aligned
    assert torch.equal(ops.bsi_layer_forward(x.view(1, Q, D), keys, bias, 2), want.view(1, Q, R))


# 32 MB of keys: beyond 32 groups the rows are packed by a launch of their own
def test_one_launch_rule_at_large_key_sets():
    fits = capi.lib().bsi_b200_linear_decode_fits
    assert [fits(2, 8192, 4096), fits(3, 8192, 4096), fits(8, 8191, 4096), fits(9, 8191, 4096)] == [1, 0, 1, 0]
    x, k = _inputs.fc1(Q=3, R=8192, D=4096, seed=3, dtype=torch.float32)
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    both = ops.bsi_layer_forward(x.to(DEV), keys, None, 2)
    assert torch.equal(both[:2], ops.bsi_layer_forward(x[:2].to(DEV), keys, None, 2))


# a single row has any row stride: a transposed column (1), one of several columns, a broadcast row (0), the last of many
@pytest.mark.parametrize("D,R", [(512, 300), (16384, 8192)])
def test_one_row_of_any_row_stride(D, R):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    x, k = _inputs.fc1(Q=1, R=R, D=D, seed=D, dtype=torch.float32)
    x = x.to(DEV)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    want = ops.bsi_layer_forward(x.clone(), keys, None, 2)
    column = x.clone().view(D, 1)
    assert column.t().stride() == (1, 1)
    for row in (column.t(), torch.cat([column, column], 1)[:, 1:].t(), x.view(1, 1, D).expand(1, 1, D),
                x.as_strided((1, D), (0, 1)), torch.cat([x + 1.0, x])[1:], x.as_strided((1, D), (1 << 40, 1))):
        for call in (ops.bsi_layer_forward, lambda *a: ops.bsi_linear_forward(a[0].reshape(1, D), *a[1:])):
            assert torch.equal(call(row, keys, None, 2).view(1, R), want)


# a pinned tensor-core engine holds for layers of few rows too: the tiles count themselves, the key-streaming kernel does not
def test_pinned_engine_is_not_replaced(monkeypatch):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    x, k = _inputs.c1(Q=8, R=300, D=512)
    x = x.to(DEV)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    packed = torch.empty(8, 512, dtype=torch.int8, device=DEV), torch.empty(8, 2, device=DEV)
    ops.pack_queries_into(x, *packed, 2)
    calls = (lambda: ops.bsi_layer_forward(x, keys, None, 2), lambda: ops.linear_from_packed(*packed, keys, None, 2, torch.float32))
    for call in calls:
        capi.exact_int_tiles()
        free = call()
        assert capi.exact_int_tiles() == 0
        monkeypatch.setenv("BSI_B200_ENGINE", "tcgen05")
        pinned = call()
        monkeypatch.delenv("BSI_B200_ENGINE")
        assert capi.exact_int_tiles() > 0 and torch.equal(free, pinned)


# the profile of the last build is that of the last call: a one-launch layer has none
def test_one_launch_layer_leaves_no_old_profile(monkeypatch):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    x, k = _inputs.c1(Q=8, R=300, D=512)
    x = x.to(DEV)
    keys = ops.build_bsi_keys_cuda(k.to(DEV), 2)[0]
    monkeypatch.setenv("BSI_PROFILE", "1")
    ops.bsi_linear_forward(x, keys, None, 2)
    assert ops.get_last_query_build_profile_cuda()[2] > 0
    monkeypatch.delenv("BSI_PROFILE")
    ops.bsi_linear_forward(x, keys, None, 2)
    assert ops.get_last_query_build_profile_cuda() == (0, 0, 0)


# The kernel may read keys ahead of the kernel before it only once the host has seen the key set's build done; a call right
# behind the build, or recorded in a graph, does not count as having seen it.
@pytest.mark.parametrize("Q", [4, 16])
def test_keys_count_as_complete_only_when_seen(Q):
    import bsipytorch_b200
    ops = bsipytorch_b200.bsi_ops
    x, k = _inputs.fc1(Q=Q, R=700, D=4096, seed=Q, dtype=torch.float32)
    x, k = x.to(DEV), k.to(DEV)
    want = ops.bsi_layer_forward(x, ops.build_bsi_keys_cuda(k, 2)[0], None, 2)
    complete = lambda keys: ops.debug_keys_tensors(keys)["complete"]      # noqa: E731
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)
    keys = ops.build_bsi_keys_cuda(k, 2)[0]
    passes = [ops.bsi_layer_forward(x, keys, None, 2) for _ in range(3)]
    assert not complete(keys)
    torch.cuda.synchronize()
    passes.append(ops.bsi_layer_forward(x, keys, None, 2))
    assert complete(keys)
    assert all(torch.equal(y, want) for y in passes)
    keys = ops.build_bsi_keys_cuda(k, 2)[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = ops.bsi_layer_forward(x, keys, None, 2)
    assert not complete(keys)
    graph.replay()
    assert torch.equal(captured, want)
    queries = ops.build_bsi_queries_cuda_batch_packed(x, 2)
    for _ in range(3):
        assert torch.equal(ops.batch_dot_product_multiquery_cuda_batch_caps(queries, keys)[0], want)
        torch.cuda.synchronize()
    with torch.cuda.graph(torch.cuda.CUDAGraph()):                        # the question may be asked inside a capture
        ops.bsi_layer_forward(x, keys, None, 2)
    assert complete(keys)
