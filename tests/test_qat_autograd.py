"""The training step of ``Linear`` as a node of autograd: failures, saved tensors and derivatives of its gradients."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def Linear(lib_built):
    from t81lib_b200 import _capi
    from t81lib_b200.nn import Linear
    assert _capi.device_available(), _capi.last_error()
    return Linear


def test_a_library_error_in_the_backward_is_raised(Linear):
    layer = Linear(96, 64, bias=False, device="cuda").train()
    x = torch.randn(20, 96, device="cuda")
    # a hook that hands the saved input back in a type the weight gradient refuses, on the host and before any launch
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.double() if t.shape == x.shape else t):
        y = layer(x)
    with pytest.raises(ValueError, match="operand dtypes"):
        y.sum().backward()
    layer(x).sum().backward()  # and the next step is none the worse
    assert layer.weight.grad.isfinite().all()


def _twins(Linear, shape, dtype=torch.float32):
    """The same layer on the device and in its PyTorch form on the CPU, and an input for each."""
    torch.manual_seed(7)
    layer, twin = Linear(48, 32, device="cuda").train(), Linear(48, 32).train()
    twin.load_state_dict({k: v.cpu() for k, v in layer.state_dict().items()}, strict=False)
    x = torch.randn(*shape, dtype=dtype)
    return ((layer, x.cuda().requires_grad_(True)), (twin, x.clone().requires_grad_(True)))


# a gradient penalty on the input and on the weight: derivatives of the step's gradients, against the PyTorch form
@pytest.mark.parametrize("shape", [(20, 48), (2, 9, 48)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_gradients_of_gradients(Linear, shape, dtype):
    results = []
    for layer, x in _twins(Linear, shape, dtype):
        if dtype == torch.float64 and not x.is_cuda:
            x = x.detach().float().requires_grad_(True)  # the device layer computes in float32
        y = torch.tanh(layer(x))
        gx, gw = torch.autograd.grad(y.sum(), [x, layer.weight], create_graph=True)
        penalty = (gx ** 2).sum() + (gw ** 2).sum()
        results.append([t.detach().cpu().double() for t in torch.autograd.grad(penalty, [x, layer.weight, layer.bias])])
    for got, want in zip(*results):
        # fp32 throughout; the device forward takes activations with 16 mantissa bits (2^-17 each)
        assert float((got - want).norm() / want.norm()) < 4 * 2.0 ** -16
        assert float(want.norm()) > 0


def test_a_batch_of_output_gradients(Linear):
    (layer, x), _ = _twins(Linear, (20, 48))
    y, v = layer(x), torch.randn(3, 20, 32, device="cuda")
    inputs = [x, layer.weight, layer.bias]
    got = torch.autograd.grad(y, inputs, v, retain_graph=True, is_grads_batched=True)
    for i in range(3):
        for a, b in zip(got, torch.autograd.grad(y, inputs, v[i], retain_graph=True)):
            assert float((a[i] - b).norm() / b.norm()) < 1e-6  # both exact products summed in fp32


def test_saved_tensors_that_come_back_otherwise(Linear):
    (layer, x), _ = _twins(Linear, (20, 48))
    v = torch.randn(20, 32, device="cuda")
    inputs = [x, layer.weight, layer.bias]
    want = torch.autograd.grad(layer(x), inputs, v)
    start = layer.training_scale.clone()
    # column by column instead of row by row
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.t().contiguous(), lambda t: t.t()):
        y = layer(x)
    assert torch.equal(layer.training_scale, start)  # the same weight: the same step
    for a, b in zip(torch.autograd.grad(y, inputs, v), want):
        assert torch.equal(a, b)
    # on another device: refused on the host
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.cpu()):
        y = layer(x)
    with pytest.raises(ValueError, match="saved tensors"):
        y.sum().backward()
    # and brought back from there
    with torch.autograd.graph.save_on_cpu():
        y = layer(x)
    for a, b in zip(torch.autograd.grad(y, inputs, v), want):
        assert torch.equal(a, b)
