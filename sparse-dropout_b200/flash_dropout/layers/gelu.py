"""GELU between SparseDrop layers, on the library's kernels (csrc/sd_gelu.cu).

Same module as ``torch.nn.GELU`` (the reference's models use it between the two DropoutMM of an MLP: eval/llm/model.py:60-69,
eval/vit/model.py:60-66).  A contiguous fp16 or bf16 CUDA tensor takes the kernels; everything else (CPU, fp32, the tanh form,
tracing, function transforms, forward-mode differentiation) goes to ``F.gelu``.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from flash_dropout import _lib


class GELU(torch.nn.GELU):
    """Drop-in ``torch.nn.GELU`` that takes the fused path on CUDA (see the module docstring)."""

    def forward(self, input: torch.Tensor) -> torch.Tensor:
        if input.is_cuda and self.approximate == "none" and not torch.jit.is_tracing() and not torch.compiler.is_compiling():
            y = _lib.ext().gelu(input)
            if y is not None:
                return y
        return F.gelu(input, approximate=self.approximate)
