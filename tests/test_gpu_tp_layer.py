"""The one-rank tensor-parallel decoder takes residual sums in epilogues only where that makes no difference to its caller: residual
streams of other layouts and types, modes, gradients and a user's own device operations."""
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from bsipytorch_b200 import bsi_ops, opt
from bsipytorch_b200.opt_tp import BsiDeviceOps, build_opt_tp

pytestmark = pytest.mark.gpu
DEV = "cuda"
CFG = opt.OPTConfig(vocab_size=512, hidden_size=512, num_hidden_layers=2, num_attention_heads=8, ffn_dim=2048,
                    max_position_embeddings=128, name="tiny512")
B, T = 4, 32


class _Own(BsiDeviceOps):
    """Operations with the signatures a user's subclass had before sums of squares went with them."""

    def pack_into(self, x2d, q8, scales):
        self.m.pack_queries_into(x2d, q8, scales, self.dp)

    def linear(self, q8, scales, keys, bias, out_dtype, relu=False):
        return self.m.linear_from_packed(q8, scales, keys, bias, self.dp, out_dtype, relu)

    def linear_scaled(self, q8, scales, keys, bias, out_dtype, columns, factor):
        return self.m.linear_from_packed(q8, scales, keys, bias, self.dp, out_dtype, False, columns, factor)

    def linear_requant(self, q8, scales, keys, bias, layer_dtype, relu, q8_ptrs, ld8, scale_ptrs, scale_ld):
        self.m.linear_from_packed_requant(q8, scales, keys, bias, self.dp, layer_dtype, relu, q8_ptrs, ld8, scale_ptrs, scale_ld)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@torch.no_grad()
def test_own_operations(dtype):
    ids = torch.randint(0, 512, (B, T), device=DEV)
    want = build_opt_tp(CFG, dtype=dtype, device=DEV, seed=3)(ids)
    assert torch.equal(build_opt_tp(CFG, dtype=dtype, device=DEV, seed=3, ops=_Own())(ids), want)


class _CountAdds(TorchDispatchMode):
    n = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.n += func in (torch.ops.aten.add.Tensor, torch.ops.aten.add_.Tensor)
        return func(*args, **(kwargs or {}))


class _CountFunctions(TorchFunctionMode):
    n = 0

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.n += func in (torch.Tensor.add, torch.add, torch.Tensor.__add__)
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("mode", [_CountAdds, _CountFunctions])
@torch.no_grad()
def test_modes_see_the_sums(mode):
    ids, seen = torch.randint(0, 512, (B, T), device=DEV), []
    for ops in (_Own(), None):
        model = build_opt_tp(CFG, dtype=torch.float16, device=DEV, seed=3, ops=ops)
        logits = model(ids)
        with mode() as counted:
            got = model(ids)
        assert torch.equal(got, logits)
        seen.append(counted.n)
    assert seen[0] == seen[1] >= 2 * CFG.num_hidden_layers


@torch.no_grad()
def test_matrix_to_add_in_the_epilogue_or_behind():
    Q, D, R = 40, 512, 264
    g = torch.Generator(device=DEV).manual_seed(1)
    x, add = torch.randn(Q, D, generator=g, device=DEV), torch.randn(Q, R, generator=g, device=DEV).half()
    keys = bsi_ops.build_bsi_keys_cuda(torch.randn(R, D, generator=g, device=DEV) * 0.02, 2, 0.5)[0]
    q8, sc = torch.empty(Q, D, dtype=torch.int8, device=DEV), torch.empty(Q, D // 256, device=DEV)
    bsi_ops.pack_queries_into(x, q8, sc, 2)
    y = bsi_ops.linear_from_packed(q8, sc, keys, None, 2, torch.float16)
    wide, odd = torch.empty(Q, 2 * R, dtype=torch.float16, device=DEV), torch.empty(Q * R + 1, dtype=torch.float16, device=DEV)
    wide[:, :R] = add
    odd[1:] = add.view(-1)
    for a in (add, wide[:, :R], add.t().contiguous().t(), odd[1:].view(Q, R), add.float(), add.bfloat16(), add[:1].expand(Q, R)):
        got = bsi_ops.linear_from_packed(q8, sc, keys, None, 2, torch.float16, add=a)
        assert got.dtype == (a + y).dtype and torch.equal(got, a + y)
    with torch.enable_grad():
        leaf = add.clone().requires_grad_(True)
        assert bsi_ops.linear_from_packed(q8, sc, keys, None, 2, torch.float16, add=leaf).grad_fn is not None
    with _CountAdds() as counted:
        assert torch.equal(bsi_ops.linear_from_packed(q8, sc, keys, None, 2, torch.float16, add=add), add + y)
    assert counted.n == 2


def test_matrices_that_cannot_be_added_are_refused():
    keys = bsi_ops.build_bsi_keys_cuda(torch.randn(256, 512), 2, 0.5)[0]
    q8, sc = torch.zeros(16, 512, dtype=torch.int8, device=DEV), torch.ones(16, 2, device=DEV)
    for add in (torch.zeros(16, 255, device=DEV).half(), torch.zeros(1, 256, device=DEV).half(), torch.zeros(16, 256).half(),
                torch.zeros(4096, device=DEV).half(), torch.zeros(16, 256, dtype=torch.int32, device=DEV)):
        with pytest.raises(RuntimeError, match="add must be"):
            bsi_ops.linear_from_packed(q8, sc, keys, None, 2, torch.float16, add=add)
