"""LayerNorm in front of SparseDrop layers, on the library's two HBM-bound kernels.

Same module as ``torch.nn.LayerNorm`` (same parameters and ``state_dict`` keys; the reference's models use
``nn.LayerNorm`` in front of their DropoutMM layers: eval/llm/model.py:72-74,113, eval/vit/model.py:11,53,106-108).
On a CUDA fp32 input whose normalised width is a multiple of 4 up to 1024 the forward is one pass that writes its
result in the dtype the consumer reads (the autocast dtype when autocast is on, so the separate cast disappears) and
the backward one pass for dx plus a small reduction for the parameter gradients; everything else (CPU tensors, other
dtypes, wider rows, several normalised dimensions, a trace being recorded) goes to ``F.layer_norm`` unchanged.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from flash_dropout import _lib


def layer_norm(x: torch.Tensor, normalized_shape, weight, bias, eps: float) -> torch.Tensor:
    """``F.layer_norm`` with the fused path where it applies (see the module docstring)."""
    if len(normalized_shape) == 1 and weight is not None and x.is_cuda and not torch.jit.is_tracing():
        y = _lib.ext().layer_norm(x, weight, bias, eps)       # csrc/sd_torch.cpp: forward launch and autograd node
        if y is not None:
            return y
    return F.layer_norm(x, normalized_shape, weight, bias, eps)


class LayerNorm(torch.nn.LayerNorm):
    """Drop-in ``torch.nn.LayerNorm`` that takes the fused path on CUDA (see the module docstring)."""

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        return layer_norm(input, self.normalized_shape, self.weight, self.bias, self.eps)
