"""train-gpt's `losses.py` on the CUDA path: the capped-logit cross-entropy and its gradient from
one pass over the logits.

The reference computes `cross_entropy_loss(params, input_ids, target_ids, cfg)` as
`forward(...)` (which ends with `cap * tanh(logits / cap)`, model.py:97), a float32 cast,
`log_softmax`, a gather and a mean (losses.py:8-12).  Here the part after the unembedding
GEMM is `capped_cross_entropy(logits, target_ids, cap)`: it takes the GEMM's raw bf16 output,
so the capped logits and their float32 copy are never written to memory.
"""
from __future__ import annotations

import torch

from . import ops


def capped_cross_entropy(logits: torch.Tensor, target_ids: torch.Tensor, cap: float) -> torch.Tensor:
    """Mean over tokens of -log_softmax(cap * tanh(logits / cap))[target] (model.py:97, losses.py:8-12).

    logits: (..., vocab) bf16, the unembedding GEMM's output BEFORE the cap; target_ids: (...)
    integer.  Any vocabulary size (the reference's default 50257 is not a multiple of 8).
    Differentiable with respect to logits.

    With gradients on and logits that require one, the FORWARD writes the gradient too (for an upstream
    gradient of 1; another one is seen in the backward pass and the gradient made again from the logits): one
    read of the logits serves both.  The logits and a tensor of their size stay allocated until the backward pass
    or the result's end, and a loss that is never differentiated pays for the write: 8192 x 50257 359 us with it,
    230 under `torch.no_grad()`.  (A vocabulary or cap that a row in shared memory cannot hold
    takes two passes, which keep one tensor of that size.)"""
    return ops._host().capped_cross_entropy(logits, target_ids, cap)
