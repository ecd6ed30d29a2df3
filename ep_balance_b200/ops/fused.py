"""Autograd wrappers of the dense models' native kernels.

Each public function takes the native path for the tensors its kernels cover and the PyTorch formulation for everything
else (other devices, types, alignments, function transforms and forward-mode AD, which a custom autograd function has
no rule for).
"""

from __future__ import annotations

import torch
import torch.nn.functional as F
from torch.autograd import forward_ad
from torch.autograd.function import once_differentiable

from .extension import load


def plain_autograd() -> bool:
    """No function transform (vmap, grad, jvp) and no forward-mode level is active."""
    return not torch._C._are_functorch_transforms_active() and forward_ad._current_level < 0


class _TokenCrossEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets):
        log_prob = torch.log_softmax(logits.float(), -1)
        loss, weight = torch.ops.aten.nll_loss_forward(log_prob, targets, None, 1, -100)  # 1: mean
        ctx.save_for_backward(log_prob, targets, weight)
        return loss

    @staticmethod
    @once_differentiable
    def backward(ctx, dloss):
        log_prob, targets, weight = ctx.saved_tensors
        grad = torch.empty_like(log_prob, dtype=torch.bfloat16)
        load().cross_entropy_backward(log_prob, targets, weight, dloss.contiguous(), grad)
        return grad, None


def token_cross_entropy(logits: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
    """``F.cross_entropy(logits.float(), targets)`` for ``logits`` [rows, vocab] and ``targets`` [rows] (mean over the rows whose
    target is not -100), with the gradient of bf16 logits on a GPU taken from the log-probabilities in one pass."""
    if (logits.is_cuda and logits.dtype == torch.bfloat16 and targets.dtype == torch.int64 and targets.device == logits.device
            and logits.dim() == 2 and targets.shape == logits.shape[:1] and logits.shape[0] > 0 and logits.shape[1] % 8 == 0
            and logits.is_contiguous() and logits.data_ptr() % 16 == 0 and plain_autograd()):
        return _TokenCrossEntropy.apply(logits, targets.contiguous())
    return F.cross_entropy(logits.float(), targets)
