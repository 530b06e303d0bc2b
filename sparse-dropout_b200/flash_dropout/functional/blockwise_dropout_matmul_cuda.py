"""SparseDrop linear on the sm_100a kernels: the entry point of the operator API.

Same contract as the reference's ``BlockwiseDropoutMatmulCUDA``
(flash_dropout/functional/blockwise_dropout_matmul_cuda.py:7-59): forward ``y = (keep o x) W^T / (1-p)``
by a DSD product, backward ``dx`` by an SDD product and ``dW`` by a DSD product over the transposed
operands.  Differences: the mask comes from the device-side Philox plan kernel instead of
``torch.rand`` (one launch, no host sync, and the same plan is reused by all three products);
bf16 is accepted as well as fp16; launches go to the current stream of the tensors' device.

The checks, casts, launches and the autograd node are native code (``csrc/sd_torch.cpp``: ``linear``,
``SparseDropLinearBackward``); this file chooses the mask and hands over.
"""
from __future__ import annotations

import weakref

import torch

from flash_dropout import _lib
from flash_dropout import random as sd_random
from flash_dropout.cuda.binding_gemm import BlockPlan, PlanBatch, _rep

from .recorded import recorded

_last_cast = {"key": None, "src": None, "ref": None}


def _autocast_input(input: torch.Tensor, dt: torch.dtype) -> torch.Tensor:
    """``input.to(dt)``, shared between consecutive calls with the very same tensor: one cast for the q / k / v projections
    of an attention block, and one cast of the summed gradient backward.

    For callers that know that nothing but torch operators writes ``input``.  The operators cast for themselves instead: a
    CUDA graph's replay rewrites tensors without advancing their version, and a copy made during a capture holds nothing
    before the first replay.

    The entry is valid only for the very tensor it was made from, unmodified since.  The tensor is identified by the object
    that owns its memory (a view's base) plus the view's geometry; the entry holds only a weak reference to that owner, so
    once it is freed the entry is dead and a new tensor that the allocator places at the same address can never be taken
    for it."""
    if input.dtype == dt:
        return input
    owner = input._base if input._base is not None else input
    key = (input._version, tuple(input.shape), tuple(input.stride()), input.storage_offset(), input.dtype, dt,
           input.requires_grad, torch.is_grad_enabled())
    src = _last_cast["src"]
    if src is not None and src() is owner and _last_cast["key"] == key:
        cached = _last_cast["ref"]()
        if cached is not None:
            return cached
    out = input.to(dt)
    _last_cast["key"], _last_cast["src"], _last_cast["ref"] = key, weakref.ref(owner), weakref.ref(out)
    return out


def blockwise_dropout_matmul(input: torch.Tensor, weight: torch.Tensor, block_size: int, p: float,
                             plan: BlockPlan | None = None, relu: bool = False, input_relu: bool = False,
                             grad_premasked: bool = False, wgrad=None, recompute_plan: bool = False,
                             weight_lowp: torch.Tensor | None = None, any_rank: bool = False) -> torch.Tensor:
    """``y = (mask o input) . weight^T / (1 - p)`` with a fresh block mask (or the given plan).

    Under CUDA autocast both operands are cast to the autocast dtype (the reference casts to fp16,
    blockwise_dropout_matmul_cuda.py:9); otherwise they must already be fp16 or bf16.  fp32 operands get their
    gradients in fp32 straight from the kernels.  The keyword arguments after ``plan`` fuse elementwise neighbours into
    the kernels' epilogues (all off by default):
      relu            the result goes through ReLU in the forward epilogue (eval/mlp/model.py:33-38 applies it as a
                      separate op after every layer);
      input_relu      ``input`` is the output of a ReLU: the dX epilogue multiplies by its derivative (input > 0), so
                      the gradient this layer returns is already the gradient of the ReLU's input;
      grad_premasked  with ``relu``: the incoming gradient already carries this layer's ReLU derivative (its only
                      consumer is a layer called with ``input_relu``), so backward does not apply it again;
      wgrad           ``(tensor [out, in], accumulate, notify)``: the weight gradient is written (or, in fp32, added)
                      straight into that tensor, fp32 or of the operands' type, by the dW epilogue instead of being
                      returned to autograd; ``notify()`` is called afterwards;
      recompute_plan  keep only (seed, offset) of the mask between forward and backward and draw the plan again there
                      (one more plan launch per layer in backward; the plan buffer, 4 bytes per tile and list entry, is
                      not kept alive).  Applies to plans drawn from a host-side offset, a given one with the block size
                      and p it was drawn with; a plan whose offset was read from the device-side counter (CUDA-graph
                      mode, where plan buffers are static anyway) is kept;
      weight_lowp     an up-to-date copy of ``weight`` in the autocast dtype that the caller keeps (a training step that
                      casts all weights with one launch): used instead of casting again, which needs ``wgrad`` (the copy
                      is outside autograd, so the weight gradient has to leave through the fused store);
      any_rank        ``input`` may have any number of leading dimensions, all of them rows.
    """
    assert 0 <= p < 1, "Dropout probability must be in [0, 1)"
    if torch.jit.is_tracing():
        return recorded(blockwise_dropout_matmul, (input, weight), block_size, p, plan, relu, input_relu, grad_premasked, wgrad,
                        recompute_plan, None, any_rank)
    rep_r, rep_c = _rep(block_size)
    draw_p = p
    seed = offset = 0
    counter = None
    fresh = False
    if plan is None:
        if PlanBatch.active is not None:
            K = input.shape[-1]
            plan = BlockPlan.draw(input.numel() // K, K, block_size, p, input.device)
        elif input.is_cuda and (counter := sd_random.device_counter(input.device)) is not None:
            seed, offset = sd_random.seed_and_base()
        else:
            seed, offset = sd_random.next_seed_offset()
            fresh = True
    if plan is None:
        buf, R, C = None, 0, 0
    else:
        buf, R, C = plan.buf, plan.R, plan.C
        if recompute_plan and plan.origin is not None:
            # backward draws this very plan again, whatever block size and p the call names
            _, _, block_size, draw_p, seed, offset = plan.origin
            rep_r, rep_c = _rep(block_size)
            seed, offset = seed & (2**64 - 1), offset & (2**64 - 1)
        else:
            recompute_plan = False
    if torch.is_autocast_enabled("cuda"):
        # fp32 operands are cast inside the operator; others by autograd
        dt = torch.get_autocast_dtype("cuda")
        if input.dtype not in (dt, torch.float32):
            input = input.to(dt)
    target, accumulate, notify = wgrad if wgrad is not None else (None, False, None)
    try:
        return _lib.ext().linear(input, weight, buf, R, C, rep_r, rep_c, not isinstance(block_size, int), p, seed, offset,
                                counter, relu, input_relu, grad_premasked, target, accumulate, notify, recompute_plan,
                                weight_lowp, any_rank, draw_p)
    except Exception:
        if fresh:
            sd_random.give_back(offset)        # a call that was refused has used no mask
        raise


class BlockwiseDropoutMatmulCUDA:
    """The reference's name for the operator: ``BlockwiseDropoutMatmulCUDA.apply(input, weight, block_size, p)``."""

    apply = staticmethod(blockwise_dropout_matmul)
