"""The decoder layer as one extension call against the same modules called one by one: same bits, same counters."""
import pytest
import torch

from bsipytorch_b200 import opt

pytestmark = pytest.mark.gpu


# few tokens (one-launch linears), a ragged count, a full batch
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,T", [(1, 5), (3, 37), (2, 128)])
def test_native_layer_equals_module_calls(dtype, B, T):
    cfg = opt.OPTConfig(vocab_size=500, hidden_size=512, num_hidden_layers=1, num_attention_heads=8, ffn_dim=1280, name="small")
    layer = opt.build_opt_bsi(cfg, dtype=dtype, seed=3).model.decoder.layers[0]
    x = torch.randn(B, T, 512, generator=torch.Generator().manual_seed(T)).to(dtype).cuda()
    with torch.no_grad():
        assert layer._native(x) is not None
        before = layer.fc1.dot_output_elements_total
        got = layer(x)
        assert layer.fc1.dot_output_elements_total - before == B * T * 1280
        hook = layer.fc2.register_forward_hook(lambda m, a, y: None)       # somebody looks in between: module by module
        assert layer._native(x) is None
        want = layer(x)
        hook.remove()
    assert torch.equal(got, want)
