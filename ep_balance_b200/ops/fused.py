"""Autograd wrappers of the dense models' native kernels.

Each public function takes the native path for the tensors its kernels cover and the PyTorch formulation for everything
else: other devices, types and alignments, and whoever has to see the operations themselves (:func:`eager`).
"""

from __future__ import annotations

import torch
import torch.nn.functional as F
from torch.autograd import forward_ad
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext
from torch.utils._python_dispatch import is_in_torch_dispatch_mode

from .extension import load


def eager(*tensors: torch.Tensor) -> bool:
    """Plain tensors, executed now, with nobody watching.  A kernel launched through the extension is invisible to PyTorch:
    a tracer (``jit.trace``, ``make_fx``, ``compile``, ``export``) would record the allocation of its output and nothing
    that fills it, a dispatch or function mode would miss it, a subclass (a fake tensor, an fx proxy) has no memory to run
    it on, and function transforms and forward-mode AD have no rule for it.  All of them get the PyTorch operations."""
    return (not torch.compiler.is_compiling() and not torch.jit.is_tracing()
            and all(type(t) in (torch.Tensor, torch.nn.Parameter) for t in tensors)
            and torch._C._len_torch_dispatch_stack() == 0 and not is_in_torch_dispatch_mode()
            and (torch._C._len_torch_function_stack() == 0  # `with torch.device(...)` is a function mode that only sets defaults
                 or all(type(m) is DeviceContext for m in _get_current_function_mode_stack()))
            and not torch._C._are_functorch_transforms_active() and forward_ad._current_level < 0)


class _TokenCrossEntropy(torch.autograd.Function):
    """(loss, log-probabilities).  The second output is there for second derivatives: backward's formula reads it, and as an
    output it is connected to the logits."""

    @staticmethod
    def forward(ctx, logits, targets):
        log_prob = torch.log_softmax(logits.float(), -1)
        loss, weight = torch.ops.aten.nll_loss_forward(log_prob, targets, None, 1, -100)  # 1: mean
        ctx.save_for_backward(log_prob, targets, weight)
        ctx.set_materialize_grads(False)
        ctx.dtype = logits.dtype
        return loss, log_prob

    @staticmethod
    def backward(ctx, dloss, dlog_prob):
        log_prob, targets, weight = ctx.saved_tensors
        if dlog_prob is None and not torch.is_grad_enabled() and eager(log_prob, targets, dloss):
            grad = torch.empty_like(log_prob, dtype=torch.bfloat16)
            load().cross_entropy_backward(log_prob, targets, weight, dloss.contiguous(), grad)
            return grad, None
        prob = log_prob.exp()
        grad = torch.zeros_like(prob)
        if dloss is not None:
            counted = targets != -100
            scale = torch.where(counted, dloss / weight, 0.0).unsqueeze(1)
            grad = (prob * scale).scatter_add(1, torch.where(counted, targets, 0).unsqueeze(1), -scale)
        if dlog_prob is not None:
            grad = grad + dlog_prob - prob * dlog_prob.sum(-1, keepdim=True)
        return grad.to(ctx.dtype), None


def token_cross_entropy(logits: torch.Tensor, targets: torch.Tensor) -> torch.Tensor:
    """``F.cross_entropy(logits.float(), targets)`` for ``logits`` [rows, vocab] and ``targets`` [rows] (mean over the rows whose
    target is not -100), with the gradient of bf16 logits on a GPU taken from the log-probabilities in one pass."""
    if (eager(logits, targets) and logits.is_cuda and logits.dtype == torch.bfloat16 and targets.dtype == torch.int64
            and targets.device == logits.device and logits.dim() == 2 and targets.shape == logits.shape[:1]
            and logits.shape[0] > 0 and logits.shape[1] % 8 == 0 and logits.is_contiguous() and logits.data_ptr() % 16 == 0):
        return _TokenCrossEntropy.apply(logits, targets.contiguous())[0]
    return F.cross_entropy(logits.float(), targets)


def _dense_heads(g: torch.Tensor) -> torch.Tensor:
    ok = g.dtype == torch.bfloat16 and g.stride(3) == 1 and g.data_ptr() % 16 == 0 and all(s % 8 == 0 for s in g.stride()[:3])
    return g if ok else g.to(torch.bfloat16).contiguous(memory_format=torch.contiguous_format).clone()


def _rotate_back(g, cos, sin):
    g1, g2 = g[..., : g.shape[-1] // 2], g[..., g.shape[-1] // 2:]
    return torch.cat([g1 * cos + g2 * sin, g2 * cos - g1 * sin], dim=-1)


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
    def backward(ctx, dq, dk, dv):
        cos, sin = ctx.saved_tensors
        if torch.is_grad_enabled() or not eager(dq, dk, dv, cos, sin):  # second derivatives: the operations themselves
            back = _rotate_back(dq, cos, sin), _rotate_back(dk, cos, sin), dv
            return torch.stack([g.transpose(1, 2) for g in back], 2), None, None
        dqkv = torch.empty(ctx.shape, dtype=torch.bfloat16, device=cos.device)
        load().rope(dqkv, _dense_heads(dq), _dense_heads(dk), _dense_heads(dv), cos, sin, True)
        return dqkv, None, None


def split_rotate(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """``qkv`` [B, S, 3, heads, dim] -> q and k with rotary embedding in one kernel, and v (a view), each
    [B, heads, S, dim]; None where the kernel does not apply.  ``cos`` / ``sin``: [S, dim / 2] tables without gradients."""
    if not eager(qkv, cos, sin):
        return None
    tables = all(t.dtype == torch.bfloat16 and t.device == qkv.device and t.is_contiguous() and t.data_ptr() % 16 == 0
                 and t.shape == (qkv.shape[1], qkv.shape[4] // 2) and not t.requires_grad for t in (cos, sin))
    if (tables and qkv.is_cuda and qkv.dtype == torch.bfloat16 and qkv.is_contiguous() and qkv.data_ptr() % 16 == 0
            and qkv.shape[4] % 16 == 0 and qkv.numel() > 0):
        return _SplitRotate.apply(qkv, cos, sin)
    return None


def _plain_bf16(*tensors: torch.Tensor) -> bool:
    """No autograd on any of them, and vectors of eight bf16 values at 16-byte addresses on one GPU."""
    return (eager(*tensors) and not torch.is_grad_enabled() and not torch.is_autocast_enabled("cuda")
            and all(t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous() and t.numel() > 0 and t.data_ptr() % 16 == 0
                    and t.device == tensors[0].device for t in tensors))


def swiglu(packed: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up`` of ``packed`` [..., 2F] = (gate, up); one kernel where autograd is off (the same bits)."""
    if not torch.jit.is_scripting():
        if _plain_bf16(packed) and packed.dim() == 2 and packed.shape[1] % 16 == 0:
            out = packed.new_empty((packed.shape[0], packed.shape[1] // 2))
            load().swiglu(packed, out)
            return out
    gate, up = packed.chunk(2, dim=-1)
    return F.silu(gate) * up


def add3(a: torch.Tensor, b: torch.Tensor, c: torch.Tensor) -> torch.Tensor:
    """``a + b + c``; one kernel where autograd is off (the same bits)."""
    if not torch.jit.is_scripting():
        if _plain_bf16(a, b, c) and a.shape == b.shape == c.shape and a.numel() % 8 == 0:
            out = torch.empty_like(a)
            load().add3(a, b, c, out)
            return out
    return a + b + c
