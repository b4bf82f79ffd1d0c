"""Sums of squares handed to the re-quantising linear go with that call alone: what the caller has registered for the same packed
activations is there afterwards, and the integers are those of the call without them."""
import pytest
import torch

import _capi_helpers as H
import _inputs
from bsipytorch_b200 import bsi_ops, capi
from oracle import oracle as o

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_registered_bounds_outlive_the_call(dtype):
    Q, R, D = 512, 1024, 2048
    chunks, tiles = D // 256, 2 * 4 * 16          # tiles of 256 x 256, 16 epilogue warps each
    q, k = _inputs.fc1(Q=Q, R=R, D=D, dtype=dtype)
    q8, scales, sq = (torch.empty(Q, D, dtype=torch.int8, device=DEV), torch.empty(Q, chunks, device=DEV), torch.empty(Q, chunks, device=DEV))
    bsi_ops.pack_queries_into(q.to(DEV), q8, scales, 2, sq)
    keys = bsi_ops.build_bsi_keys_cuda(k, 2, 0.5)[0]
    kb = H.quantize_pack(k.to(DEV), 2, 6, False)
    bounds = torch.empty(3, R, device=DEV)
    L = capi.lib()
    capi.check(L.bsi_b200_key_bounds(capi.ptr(kb["q8"]), D, R, chunks, capi.ptr(bounds), capi.stream_ptr()))

    def requant(norms):
        r8, rs = torch.full((Q, R), 99, dtype=torch.int8, device=DEV), torch.full((Q, R // 256), -1.0, device=DEV)
        capi.exact_int_tiles()
        bsi_ops.linear_from_packed_requant(q8, scales, keys, None, 2, dtype, True, [r8.data_ptr()], R, [rs.data_ptr()], R // 256, norms)
        return r8, rs, capi.exact_int_tiles()

    def whole_dot():
        capi.exact_int_tiles()
        H.dot_i8(q8, scales, kb["q8"], kb["scales"], o.scale_inv(2), 3256)
        return capi.exact_int_tiles()

    without = requant(None)
    given = requant(sq)
    assert without[2] < given[2] == tiles         # the sums arrive
    assert torch.equal(without[0], given[0]) and torch.equal(without[1], given[1])
    own = sq.clone()
    capi.check(L.bsi_b200_register_key_bounds(capi.ptr(kb["q8"]), capi.ptr(bounds), R, 64))
    capi.check(L.bsi_b200_register_query_bounds(capi.ptr(q8), capi.ptr(own), chunks))
    try:
        assert whole_dot() == tiles
        requant(sq)
        assert whole_dot() == tiles
        assert requant(None)[2] == tiles          # a call without its own reads the registered ones, as before
    finally:
        capi.check(L.bsi_b200_unregister_key_bounds(capi.ptr(kb["q8"])))
        capi.check(L.bsi_b200_unregister_query_bounds(capi.ptr(q8)))
    assert requant(None)[2] == without[2]         # nothing stays behind


def test_refusals():
    Q, R, D = 16, 256, 512
    q8, sc, keys = torch.zeros(Q, D, dtype=torch.int8, device=DEV), torch.ones(Q, 2, device=DEV), bsi_ops.build_bsi_keys_cuda(torch.randn(R, D), 2, 0.5)[0]
    x = torch.randn(Q, D, device=DEV)
    r8, rs = torch.empty(Q, R, dtype=torch.int8, device=DEV), torch.empty(Q, 1, device=DEV)
    wrong = [torch.ones(Q, 2), torch.ones(Q, 2, device=DEV).half(), torch.ones(Q, 3, device=DEV), torch.ones(2, Q, device=DEV).t()]
    for sq in wrong:
        with pytest.raises(RuntimeError, match="sq_norms"):
            bsi_ops.pack_queries_into(x, q8, sc, 2, sq)
        with pytest.raises(RuntimeError, match="sq_norms"):
            bsi_ops.linear_from_packed(q8, sc, keys, None, 2, torch.float16, sq_norms=sq)
        with pytest.raises(RuntimeError, match="sq_norms"):
            bsi_ops.linear_from_packed_requant(q8, sc, keys, None, 2, torch.float16, True, [r8.data_ptr()], R, [rs.data_ptr()], 1, sq)
