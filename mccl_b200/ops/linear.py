"""fp32 linear layer whose three products run on the tensor cores (``csrc/kernels/gemm_f32.cu``).

Same numbers as ``torch.nn.functional.linear`` in fp32, up to rounding: every product is a sum of six bf16 products
accumulated in fp32, further from no exact result than the fp32 kernels it stands in for.  Calls that the kernels do not take
(other types and devices, small products, autocast, TF32 allowed, tracing, transforms) are ``torch.nn.functional.linear``.
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

_PLAIN = (torch.Tensor, nn.Parameter)


def linear(input: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``input @ weight.T + bias``."""
    if (type(input) in _PLAIN and type(weight) in _PLAIN and (bias is None or type(bias) in _PLAIN) and input.is_cuda and not torch.compiler.is_compiling()
            and torch._C._get_tracing_state() is None and not torch._C._is_torch_function_mode_enabled()):
        from .. import require_native
        return require_native()._linear(input, weight, bias)
    return F.linear(input, weight, bias)


class Linear(nn.Linear):
    """``torch.nn.Linear`` on :func:`linear`; ``stock`` (an attribute, off) keeps torch's kernels."""

    stock: bool = False

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        if torch.jit.is_scripting():
            return F.linear(input, self.weight, self.bias)
        elif self.stock:
            return F.linear(input, self.weight, self.bias)
        else:
            return linear(input, self.weight, self.bias)
