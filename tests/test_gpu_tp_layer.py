"""The one-rank tensor-parallel decoder layer takes residual sums in epilogues only where that makes no difference to its caller:
the pair it returns, residual streams of other layouts and types, modes, gradients and hooks are those of the general form, which
a subclass of the device operations still runs."""
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from bsipytorch_b200 import bsi_ops, capi, opt
from bsipytorch_b200.opt_tp import BsiDeviceOps, build_opt_tp

pytestmark = pytest.mark.gpu
DEV = "cuda"
CFG = opt.OPTConfig(vocab_size=512, hidden_size=512, num_hidden_layers=2, num_attention_heads=8, ffn_dim=2048,
                    max_position_embeddings=128, name="tiny512")
B, T, H = 4, 32, 512


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


def _layers(dtype, cfg=CFG):
    return (build_opt_tp(cfg, dtype=dtype, device=DEV, seed=3).layers[0],
            build_opt_tp(cfg, dtype=dtype, device=DEV, seed=3, ops=_Own()).layers[0])


def _stream(dtype, rows=B * T, h=H, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(rows, h, generator=g, device=DEV).to(dtype), (torch.randn(rows, h, generator=g, device=DEV) * 0.3).to(dtype)


def _same(got, want):
    assert len(got) == len(want) == 2
    for a, b in zip(got, want):
        assert type(a) is type(b) and a.dtype == b.dtype and torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@torch.no_grad()
def test_own_operations(dtype):
    ids = torch.randint(0, 512, (B, T), device=DEV)
    want = build_opt_tp(CFG, dtype=dtype, device=DEV, seed=3)(ids)
    assert torch.equal(build_opt_tp(CFG, dtype=dtype, device=DEV, seed=3, ops=_Own())(ids), want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@torch.no_grad()
def test_pair_and_layouts(dtype):
    layer, general = _layers(dtype)
    x, d = _stream(dtype)
    wide = torch.empty(B * T, 2 * H, dtype=dtype, device=DEV)
    wide[:, :H] = x
    for delta in (None, d):
        want = general(x, delta, B, T)
        _same(layer(x, delta, B, T), want)
        _same(layer(wide[:, :H], delta, B, T), want)
        _same(layer(x.t().contiguous().t(), delta, B, T), want)
    if dtype == torch.float16:          # a wider residual stream beside 16-bit linears
        for m in (layer, general):
            m.self_attn_layer_norm.float()
            m.final_layer_norm.float()
        _same(layer(x.float(), d, B, T), general(x.float(), d, B, T))
    assert bsi_ops.device_status() == 0


# deep and narrow enough that fc2 (float32, whose packer leaves the sums of squares) is split along K
@torch.no_grad()
def test_split_dots():
    cfg = opt.OPTConfig(vocab_size=64, hidden_size=1024, num_hidden_layers=1, num_attention_heads=8, ffn_dim=8192,
                        max_position_embeddings=128, name="deep")
    layer, general = _layers(torch.float32, cfg)
    x, d = _stream(torch.float32, 80, 1024)
    want = general(x, d, 2, 40)
    _same(layer(x, d, 2, 40), want)
    assert capi.last_tiles()[1] > 1
    got = layer(x, d, 2, 40, summed=True)
    assert got[1] is None and torch.equal(got[0], want[0] + want[1])
    assert capi.last_tiles()[1] > 1


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
    layer, general = _layers(torch.float16)
    x, d = _stream(torch.float16)
    want = general(x, d, B, T)
    for m in (general, layer):
        with mode() as counted:
            got = m(x, d, B, T)
        assert counted.n == 2
        _same(got, want)
    ids, seen = torch.randint(0, 512, (B, T), device=DEV), []
    for ops in (_Own(), None):
        model = build_opt_tp(CFG, dtype=torch.float16, device=DEV, seed=3, ops=ops)
        logits = model(ids)
        with mode() as counted:
            got = model(ids)
        assert torch.equal(got, logits)
        seen.append(counted.n)
    assert seen[0] == seen[1] >= 2 * CFG.num_hidden_layers


def test_gradients_and_tangents_pass_along_the_residual_stream():
    layer, general = _layers(torch.float16)
    x, d = _stream(torch.float16)
    grads = []
    for m in (layer, general):
        leaf = x.clone().requires_grad_(True)
        y, o = m(leaf, d, B, T)
        assert y.requires_grad
        y.float().sum().backward()
        grads.append(leaf.grad)
    assert torch.equal(grads[0], grads[1]) and bool((grads[0] == 1).all())
    from torch.autograd import forward_ad as fwad
    tangents = []
    for m in (layer, general):
        with fwad.dual_level(), torch.no_grad():
            dual = fwad.make_dual(x, torch.ones_like(x))
            tangents.append(fwad.unpack_dual(m(dual, None, B, T)[0]).tangent)
    assert tangents[0] is not None and torch.equal(tangents[0], tangents[1])


@torch.no_grad()
def test_hooks_see_the_pair():
    model = build_opt_tp(CFG, dtype=torch.float16, device=DEV, seed=3)
    ids = torch.randint(0, 512, (B, T), device=DEV)
    want, seen = model.hidden_states(ids), []
    handle = model.layers[1].register_forward_hook(lambda m, args, out: seen.append((len(args), out)))
    assert torch.equal(model.hidden_states(ids), want)
    handle.remove()
    assert len(seen) == 1 and seen[0][0] == 5 and all(isinstance(t, torch.Tensor) for t in seen[0][1])
    assert torch.equal(model.final_layer_norm(seen[0][1][0] + seen[0][1][1]).view_as(want), want)


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
