"""The eval-mode forward of ``Linear`` and ``TernaryTensor`` on the routes around the native call: biases that are no plain parameter,
first calls inside a graph capture."""

import pytest
import torch
import torch.nn.utils.prune as prune
from torch.nn.utils import parametrize

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Linear(lib_built):
    from t81lib_b200 import _capi
    from t81lib_b200.nn import Linear
    assert _capi.device_available(), _capi.last_error()
    return Linear


class _Doubled(torch.nn.Module):
    def forward(self, t):
        return 2.0 * t


@pytest.mark.parametrize("change", [lambda l: prune.random_unstructured(l, "bias", 0.5),
                                    lambda l: parametrize.register_parametrization(l, "bias", _Doubled())])
def test_a_bias_that_is_no_parameter(Linear, change):
    layer = Linear(96, 64, device="cuda").eval().requires_grad_(False)
    x = torch.randn(4, 96, device="cuda")
    before, bias = layer(x), layer.bias.clone()
    change(layer)
    assert not torch.equal(layer.bias, bias)
    # fp32 sums of the same products with another last term
    torch.testing.assert_close(layer(x) - layer.bias, before - bias, rtol=0, atol=1e-5)


# A weight's first call lies inside a capture: the graph's result is right on replay, and so is a call outside the graph before it
@pytest.mark.parametrize("tokens", [4, 100, 300])
def test_first_call_inside_a_capture(lib_built, tokens):
    from t81lib_b200.torch import TernaryTensor
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    w = TernaryTensor.from_float(torch.randn(512, 768, device="cuda", generator=gen), threshold=0.45)
    x = torch.randint(-3, 4, (tokens, 768), device="cuda", generator=gen).to(torch.bfloat16)
    want = (x.double() @ w.to_trits().double().t()).float()  # whole numbers: exact in any order
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = w.matmul_input(x, out_dtype=torch.float32)
    assert torch.equal(w.matmul_input(x, out_dtype=torch.float32), want)
    y.zero_()
    graph.replay()
    assert torch.equal(y, want)


# Row scales a caller brings in another type or stride are converted, whatever the number of rows of the input
@pytest.mark.parametrize("tokens", [4, 100, 300])
@pytest.mark.parametrize("form", [lambda s: s.half(), lambda s: s.double(), lambda s: s.repeat_interleave(2)[::2]])
def test_row_scales_of_another_form(lib_built, tokens, form):
    from t81lib_b200 import ops
    from t81lib_b200.torch import TernaryTensor
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    trits = torch.randint(-1, 2, (512, 768), device="cuda", generator=gen).float()
    scale = torch.randint(1, 9, (512,), device="cuda", generator=gen).float() / 8
    packed, _ = ops.quantize_pack(trits, 0.5, "fixed")
    w = TernaryTensor(packed, (512, 768), k_actual=768, k_limbs=16, row_scale=form(scale))
    x = torch.randint(-3, 4, (tokens, 768), device="cuda", generator=gen).to(torch.bfloat16)
    want = ((x.double() @ trits.double().t()) * scale).float()  # eighths of whole numbers: exact
    assert torch.equal(w.matmul_input(x, out_dtype=torch.float32), want)
