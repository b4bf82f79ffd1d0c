"""The decoder layer as one extension call against the same modules called one by one: same bits, same counters."""
import pytest
import torch
import torch.autograd.forward_ad as forward_ad
from torch.utils._python_dispatch import TorchDispatchMode

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


def _layer(dtype=torch.float32):
    cfg = opt.OPTConfig(vocab_size=500, hidden_size=512, num_hidden_layers=1, num_attention_heads=8, ffn_dim=1280, name="small")
    layer = opt.build_opt_bsi(cfg, dtype=dtype, seed=3).model.decoder.layers[0]
    return layer, torch.randn(2, 37, 512, generator=torch.Generator().manual_seed(37)).to(dtype).cuda()


def _module_calls(layer, x):
    """The layer's modules called one by one."""
    x = x + layer.self_attn(layer.self_attn_layer_norm(x))
    return x + layer.fc2(torch.relu(layer.fc1(layer.final_layer_norm(x))))


# float32 residuals beside 16-bit attention: the sum is float32, and values beyond float16 stay finite
@pytest.mark.parametrize("low", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_layer_under_autocast_equals_module_calls(dtype, low):
    layer, x = _layer(dtype)
    if dtype == torch.float32:
        x[0, 3, 5] = 1.0e5
    with torch.no_grad(), torch.autocast("cuda", low):
        got, want = layer(x), _module_calls(layer, x)
    assert got.dtype == want.dtype and torch.equal(got, want) and bool(got.isfinite().all())


# hooks on every module see the ten modules of a layer
def test_global_hooks_fire_for_every_module():
    module = torch.nn.modules.module
    layer, x = _layer()
    for register in (module.register_module_forward_hook, module.register_module_forward_pre_hook):
        seen = []
        hook = register(lambda m, *a: seen.append(m))
        with torch.no_grad():
            layer(x)
        hook.remove()
        assert len(seen) == 10 and {id(m) for m in seen} == {id(m) for m in layer.modules()}


# wrappers that replace a module's forward on the instance
@pytest.mark.parametrize("name", ["self_attn", "self_attn_layer_norm", "self_attn.k_proj", "fc1"])
def test_forward_replaced_on_an_instance_is_called(name):
    layer, x = _layer()
    module, seen = layer.get_submodule(name), []
    own = module.forward
    module.forward = lambda x: (seen.append(1), own(x))[1]
    with torch.no_grad():
        layer(x)
    assert seen == [1]


class _Tagged(torch.Tensor):
    pass


class _Recorder(torch.overrides.TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.names.append(getattr(func, "__name__", ""))
        return func(*args, **(kwargs or {}))


def test_tensor_subclasses_and_function_modes_see_the_layer():
    layer, x = _layer()
    with torch.no_grad():
        want = layer(x)
        tagged = layer(x.as_subclass(_Tagged))
        with _Recorder() as mode:
            got = layer(x)
        with torch.device("cuda"):                 # a default device changes nothing
            assert layer._native(x) is not None
    assert type(tagged) is _Tagged and torch.equal(tagged.as_subclass(torch.Tensor), want) and torch.equal(got, want)
    assert mode.names.count("layer_norm") == 2 and "scaled_dot_product_attention" in mode.names


class _Ops(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen.append(func)
        return func(*args, **(kwargs or {}))


def test_dispatch_modes_see_the_residual_sums():
    layer, x = _layer(torch.float16)
    with torch.no_grad():
        want = layer(x)
        with _Ops() as ops:
            got = layer(x)
    assert torch.equal(got, want)
    assert ops.seen.count(torch.ops.aten.add_.Tensor) == 2


def test_residual_sums_pass_forward_tangents_on():
    layer, x = _layer()
    tangent = torch.full_like(x, 2.0)
    with torch.no_grad(), forward_ad.dual_level():
        y = forward_ad.unpack_dual(layer(forward_ad.make_dual(x, tangent)))
    assert torch.equal(y.tangent, tangent)          # the linears detach: what is left is the residual stream's


# LayerNorms without weight, without bias, over more than the last dimension, with a weight that is a buffer
@pytest.mark.parametrize("form", ["plain", "no bias", "two dimensions", "buffer"])
def test_layer_norms_of_other_forms(form):
    layer, x = _layer()
    norm = {"plain": lambda: torch.nn.LayerNorm(512, elementwise_affine=False), "no bias": lambda: torch.nn.LayerNorm(512, bias=False),
            "two dimensions": lambda: torch.nn.LayerNorm((37, 512)), "buffer": lambda: torch.nn.LayerNorm(512)}[form]().cuda()
    if form == "buffer":
        weight = norm.weight.detach() * 3.0
        del norm.weight
        norm.register_buffer("weight", weight)
    layer.final_layer_norm = norm
    with torch.no_grad():
        assert torch.equal(layer(x), _module_calls(layer, x))


def test_bias_set_as_a_parameter():
    layer, x = _layer()
    with torch.no_grad():
        want, linear = layer(x), layer.fc1(x)
        for m in (layer.self_attn.q_proj, layer.fc1):
            m.bias = torch.nn.Parameter(m.bias.clone())
        assert torch.equal(layer(x), want) and torch.equal(layer.fc1(x), linear)
        layer.fc1.fused = False
        assert torch.equal(layer.fc1(x), linear)
