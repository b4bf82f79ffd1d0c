"""The one-rank tensor-parallel decoder with device operations of a user's own."""
import pytest
import torch

from bsipytorch_b200 import opt
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
