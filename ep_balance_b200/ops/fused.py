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


def _dense_heads(g: torch.Tensor) -> torch.Tensor:
    ok = g.dtype == torch.bfloat16 and g.stride(3) == 1 and g.data_ptr() % 16 == 0 and all(s % 8 == 0 for s in g.stride()[:3])
    return g if ok else g.to(torch.bfloat16).contiguous(memory_format=torch.contiguous_format).clone()


class _SplitRotate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, cos, sin):
        B, S, _, heads, dim = qkv.shape
        q, k = (qkv.new_empty((B, heads, S, dim)) for _ in range(2))
        load().rope(qkv, q, k, None, cos, sin, False)
        ctx.save_for_backward(cos, sin)
        ctx.shape = qkv.shape
        return q, k, qkv[:, :, 2].transpose(1, 2)

    @staticmethod
    @once_differentiable
    def backward(ctx, dq, dk, dv):
        cos, sin = ctx.saved_tensors
        dqkv = torch.empty(ctx.shape, dtype=torch.bfloat16, device=cos.device)
        load().rope(dqkv, _dense_heads(dq), _dense_heads(dk), _dense_heads(dv), cos, sin, True)
        return dqkv, None, None


def split_rotate(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """``qkv`` [B, S, 3, heads, dim] -> q and k with rotary embedding in one kernel, and v (a view), each
    [B, heads, S, dim]; None where the kernel does not apply.  ``cos`` / ``sin``: [S, dim / 2] tables without gradients."""
    tables = all(t.dtype == torch.bfloat16 and t.device == qkv.device and t.is_contiguous() and t.data_ptr() % 16 == 0
                 and t.shape == (qkv.shape[1], qkv.shape[4] // 2) and not t.requires_grad for t in (cos, sin))
    if (tables and qkv.is_cuda and qkv.dtype == torch.bfloat16 and qkv.is_contiguous() and qkv.data_ptr() % 16 == 0
            and qkv.shape[4] % 16 == 0 and qkv.numel() > 0 and plain_autograd()):
        return _SplitRotate.apply(qkv, cos, sin)
    return None


def _plain_bf16(*tensors: torch.Tensor) -> bool:
    """No autograd on any of them, and vectors of eight bf16 values at 16-byte addresses on one GPU."""
    return (not torch.is_grad_enabled() and plain_autograd() and not torch.is_autocast_enabled("cuda")
            and all(type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous()
                    and t.numel() > 0 and t.data_ptr() % 16 == 0 and t.device == tensors[0].device for t in tensors))


def swiglu(packed: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up`` of ``packed`` [..., 2F] = (gate, up); one kernel where autograd is off (the same bits)."""
    f = packed.shape[-1] // 2
    if packed.dim() == 2 and packed.shape[1] % 16 == 0 and _plain_bf16(packed):
        out = packed.new_empty((packed.shape[0], f))
        load().swiglu(packed, out)
        return out
    gate, up = packed.chunk(2, dim=-1)
    return F.silu(gate) * up


def add3(a: torch.Tensor, b: torch.Tensor, c: torch.Tensor) -> torch.Tensor:
    """``a + b + c``; one kernel where autograd is off (the same bits)."""
    if a.shape == b.shape == c.shape and a.numel() % 8 == 0 and _plain_bf16(a, b, c):
        out = torch.empty_like(a)
        load().add3(a, b, c, out)
        return out
    return a + b + c
