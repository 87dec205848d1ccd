"""Ternary ``nn.Linear`` — counterpart of the reference's ``t81.nn.Linear``
(t81/nn/linear.py:18-125) with the eval forward on the B200 kernels.

Eval mode: the weight is quantised and packed once on the device
(``TernaryTensor.from_float``) and each forward is one fused kernel call —
ternary matmul, optional per-row scale, bias — on the activations where they
live.  Training mode keeps the reference's quantisation-aware forward — the
ternary quantiser with its surrogate gradient on ``weight / scale`` and a running
absmax scale (t81/nn/linear.py:72-99, t81/qat.py:12-57): with the weight on a CUDA
device the scale update, quantise + pack, the product and the gradients run on the device
kernels (``qat_linear`` of the native binding); stochastic rounding and CPU weights take the PyTorch form.
"""

from __future__ import annotations

from collections import OrderedDict
from typing import Optional

import torch
from torch import nn
from torch.nn import functional as F

from .. import _capi
from .. import torch as t81_torch

_DEFAULT_THRESHOLD = 0.45


class _StraightThrough(torch.autograd.Function):
    """Forward: the quantised values.  Backward: the gradient goes to the surrogate unchanged."""

    @staticmethod
    def forward(ctx, surrogate: torch.Tensor, quantized: torch.Tensor) -> torch.Tensor:
        return quantized

    @staticmethod
    def backward(ctx, grad_output: torch.Tensor):
        return grad_output, None


def dorso_round(x: torch.Tensor) -> torch.Tensor:
    """The surrogate whose gradient the quantiser passes on (t81/qat.py:28-34): +-1 beyond +-0.5, 2x between,
    so the weight gradient is doubled inside (-0.5, 0.5) and zero outside."""
    one = torch.ones_like(x)
    return torch.where(x >= 0.5, one, torch.where(x <= -0.5, -one, x * 2.0))


def ternary(x: torch.Tensor, threshold: float = 0.45, stochastic: bool = False) -> torch.Tensor:
    """Ternary quantiser with the reference's surrogate gradient (t81/qat.py:12-57): values are clamped to
    [-1, 1]; magnitudes at or above the threshold become their sign, the rest 0.  With ``stochastic`` a
    magnitude above the threshold survives with probability (|x| - threshold) / (1 - threshold)."""
    threshold = float(max(0.0, min(threshold, 1.0)))
    with torch.no_grad():
        clamped = x.detach().clamp(-1.0, 1.0)
        magnitude = clamped.abs()
        keep = magnitude >= threshold
        if stochastic:
            p = ((magnitude - threshold) / max(1.0 - threshold, 1e-6)).clamp(0.0, 1.0)
            keep = keep & (torch.rand_like(p) < p)
        quantized = torch.where(keep, torch.sign(clamped), torch.zeros_like(clamped))
    return _StraightThrough.apply(dorso_round(x), quantized)


class Linear(nn.Linear):
    """Balanced-ternary ``nn.Linear``; ``rule`` selects the eval-mode quantiser
    ("fixed": the reference's fixed threshold; "absmean": per-row scaled)."""

    def __init__(
        self,
        in_features: int,
        out_features: int,
        bias: bool = True,
        device: Optional[torch.device] = None,
        dtype: Optional[torch.dtype] = None,
        threshold: float = _DEFAULT_THRESHOLD,
        rule: str = "fixed",
    ) -> None:
        super().__init__(in_features, out_features, bias=bias, device=device, dtype=dtype)
        self.ternary_threshold = threshold
        self.ternary_rule = rule
        self.ternary_weight: Optional[t81_torch.TernaryTensor] = None
        self.register_buffer("training_scale", None)
        self._stochastic_rounding = False

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if self.training:
            if self.weight.is_cuda and x.is_cuda and not self._stochastic_rounding and self.weight.dtype == torch.float32:
                # fused path: running scale, quantise + pack, the product and the gradients all on the device kernels
                state = self._qat_state_on_device()
                y = _capi.native.qat_linear(x, self.weight, self.bias, state[0], 0.99, float(max(0.0, min(self.ternary_threshold, 1.0))))
                if self._buffers["training_scale"] is not state[1]:
                    self.training_scale = state[1]
                return y
            return F.linear(x, self._quantize_training_weight(), self.bias)
        ternary_weight = self.ternary_weight
        if ternary_weight is None:
            ternary_weight = self.ternary_weight = t81_torch.TernaryTensor.from_float(
                self.weight.detach(), threshold=self.ternary_threshold, rule=self.ternary_rule)
        product = ternary_weight._product
        if product is not None and t81_torch.DECODE_STREAM_LAYOUT:
            bias = self._parameters["bias"] if "bias" in self._parameters else self.bias  # past nn.Module.__getattr__ where it can be
            y = product(x, bias)  # None: a call that needs a conversion, a copy or an autograd node
            if y is not None:
                return y
        return self._packed_linear(x)

    def _packed_linear(self, x: torch.Tensor) -> torch.Tensor:
        if x.ndim == 3:
            batch, seq, features = x.shape
            return self._packed_linear(x.reshape(batch * seq, features)).reshape(batch, seq, -1)
        if x.ndim != 2:
            raise ValueError("t81.nn.Linear expects 2D or 3D inputs")
        return self.ternary_weight.matmul_input(x, bias=self.bias)

    def _quantize_training_weight(self) -> torch.Tensor:
        scale = self._update_training_scale()
        quantized = ternary(self.weight / scale, threshold=self.ternary_threshold,
                            stochastic=self._stochastic_rounding)
        return quantized * scale

    def _qat_state_on_device(self):
        """The running scale of the fused path: (four floats on the weight's device, the 0-dim view of the scale), no host
        synchronisation.  ``training_scale`` keeps its meaning (a 0-dim float32 tensor holding the running scale)."""
        device = self.weight.device
        state = self.__dict__.get("_qat_state")
        if state is None or state[0].device != device:
            values = torch.zeros(4, dtype=torch.float32, device=device)
            existing = self.training_scale
            if existing is not None:  # carried over from the PyTorch path or another device
                values[0] = existing.to(device=device, dtype=torch.float32)
                values[3] = 1.0
            state = self.__dict__["_qat_state"] = (values, values[0])
        return state

    def _update_training_scale(self) -> torch.Tensor:
        device = self.weight.device
        candidate = self.weight.detach().abs().amax().clamp(min=1e-6).to(device=device, dtype=torch.float32)
        existing = self.training_scale
        if existing is None or existing.device != device:
            self.training_scale = candidate.detach()
            return self.training_scale
        momentum = 0.99
        combined = existing.to(dtype=torch.float32) * momentum + candidate * (1.0 - momentum)
        self.training_scale = combined.clamp(min=1e-6).detach()
        return self.training_scale

    def extra_repr(self) -> str:
        base = super().extra_repr()
        if self.ternary_threshold != _DEFAULT_THRESHOLD:
            return f"{base}, threshold={self.ternary_threshold}"
        return base

    def train(self, mode: bool = True) -> "Linear":
        if mode and getattr(self, "_t81_float_released", False):
            raise RuntimeError("this layer's float weight was released at conversion; it can only run in eval mode")
        if mode:
            self.ternary_weight = None
        return super().train(mode)

    def load_state_dict(self, state_dict, strict: bool = True, assign: bool = False):
        normalized = OrderedDict()
        for key, value in state_dict.items():
            if key in {"weight", "bias"} and value.is_floating_point() and value.dtype in {torch.bfloat16, torch.float16}:
                value = value.to(torch.float32)
            normalized[key] = value
        result = super().load_state_dict(normalized, strict=strict, assign=assign)
        self.ternary_weight = None
        self.training_scale = None
        self.__dict__.pop("_qat_state", None)
        return result

    def configure_qat(self, *, stochastic_rounding: bool) -> None:
        self._stochastic_rounding = stochastic_rounding
