"""Query, key and value projections on one joint key image: same bits as one by one, and only while it is theirs."""
import pytest
import torch

import bsipytorch_b200
from bsipytorch_b200 import opt

pytestmark = pytest.mark.gpu


# few tokens (one launch), fewer than a tile, several tiles; widths of one and of several tiles per projection
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("B,T,H", [(1, 2, 256), (1, 16, 768), (2, 50, 264), (3, 100, 768)])
def test_joint_projections(dtype, B, T, H):
    cfg = opt.OPTConfig(vocab_size=300, hidden_size=H, num_hidden_layers=1, num_attention_heads=H // 64 if H % 64 == 0 else 3,
                        ffn_dim=2 * H, name="small")
    layer = opt.build_opt_bsi(cfg, dtype=dtype, seed=5).model.decoder.layers[0]
    g = torch.Generator().manual_seed(H + T)
    x = torch.randn(B, T, H, generator=g).to(dtype).cuda()
    attn = layer.self_attn
    with torch.no_grad():
        for m in (attn.q_proj, attn.k_proj, attn.v_proj):
            m.bias.copy_(torch.randn(H, generator=g) * 0.1)         # in place: the joint bias follows
        assert "_joint" in layer.__dict__
        used = bsipytorch_b200.bsi_ops.debug_joint_layers
        used()
        got = layer(x)
        assert used() == 1
        joint = layer.__dict__.pop("_joint")
        assert torch.equal(got, layer(x)) and used() == 0
        # a projection that changed its bias or its keys no longer runs on the joint image
        layer.__dict__["_joint"] = joint
        attn.k_proj.bias = attn.k_proj.bias + 1.0
        attn.v_proj._bsi_keys_cuda = bsipytorch_b200.bsi_ops.build_bsi_keys_cuda(torch.randn(H, H, generator=g) * 0.05, 2, 0.5)[0]
        changed = layer(x)
        assert used() == 0
        layer.__dict__.pop("_joint")
        assert torch.equal(changed, layer(x)) and not torch.equal(changed, got)


# replaced projections take the joint image with them (key sets loaded into a model that was built with joined ones)
def test_joint_image_goes_with_its_projections():
    cfg = opt.OPTConfig(vocab_size=300, hidden_size=1024, num_hidden_layers=1, num_attention_heads=16, ffn_dim=1024, name="small")
    layer = opt.build_opt_bsi(cfg, dtype=torch.float16, seed=5).model.decoder.layers[0]
    held = torch.cuda.memory_allocated()
    for name in ("q_proj", "k_proj", "v_proj"):
        setattr(layer.self_attn, name, torch.nn.Identity())
    words, image = 3 * 1024 * 6 * 16 * 8, 3 * 1024 * 1024
    assert held - torch.cuda.memory_allocated() >= words + image
