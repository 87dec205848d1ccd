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
