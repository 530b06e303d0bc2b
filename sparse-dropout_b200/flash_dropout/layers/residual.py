"""The residual sums around SparseDrop layers, on the library's kernel (csrc/sd_cast.cu).

``x + r`` with the stream ``x`` in fp32 and the branch ``r`` in 16 bits, as autocast leaves them (eval/llm/model.py:80-83,
eval/vit/model.py:77-80).  Contiguous CUDA tensors of one shape take the kernel; everything else is ``x + r``.
"""
from __future__ import annotations

import torch

from flash_dropout import _lib


def residual_add(x: torch.Tensor, r: torch.Tensor) -> torch.Tensor:
    if x.is_cuda and not torch.jit.is_tracing() and not torch.compiler.is_compiling():
        y = _lib.ext().residual_add(x, r)
        if y is not None:
            return y
    return x + r
