"""Second derivatives through the fused loss and rotary embedding vs the PyTorch operations they replace."""

import pytest
import torch
import torch.nn.functional as F

from ep_balance_b200.models.gpt_moe import apply_rope, rope_tables
from ep_balance_b200.ops import fused


def _penalty(f, x):
    """f, its gradient, and the gradient of the gradient's squared norm."""
    x = x.detach().requires_grad_(True)
    y = f(x)
    (g,) = torch.autograd.grad(y, x, create_graph=True)
    (h,) = torch.autograd.grad(g.float().square().sum() + y, x)
    return y.detach(), g.detach(), h


def _close(got, want):
    for a, b in zip(got, want):
        # a few bf16 roundings (2^-9 at most each), in another order
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 1.6e-2


def _loss_case(device):
    torch.manual_seed(0)
    x = (2 * torch.randn(5, 16, device=device)).bfloat16()
    return x, torch.tensor([3, -100, 0, 15, 7], device=device)


def _rope_case(device):
    torch.manual_seed(1)
    cos, sin = rope_tables(6, 16, 100.0, device, torch.bfloat16)
    return torch.randn(2, 6, 3, 2, 16, device=device).bfloat16(), cos, sin


def _mixed(parts):
    q, k, v = (p.float() for p in parts)
    return (q * k * v).sum() + (q.square() * v).sum()


def _general(qkv, cos, sin):
    q, k, v = qkv.permute(2, 0, 3, 1, 4)
    return apply_rope(q, cos, sin), apply_rope(k, cos, sin), v


def test_loss_cpu():
    x, t = _loss_case("cpu")
    _close(_penalty(lambda z: fused._TokenCrossEntropy.apply(z, t)[0], x), _penalty(lambda z: F.cross_entropy(z.float(), t), x))


def test_rotary_cpu(monkeypatch):
    class Kernels:
        @staticmethod
        def rope(qkv, q, k, v, cos, sin, backward):
            if backward:
                for i, g in enumerate((fused._rotate_back(q, cos, sin), fused._rotate_back(k, cos, sin), v)):
                    qkv[:, :, i].copy_(g.transpose(1, 2))
            else:
                for out, part in zip((q, k), _general(qkv, cos, sin)):
                    out.copy_(part)
    x, cos, sin = _rope_case("cpu")
    monkeypatch.setattr(fused, "load", lambda: Kernels)
    first = _penalty(lambda z: _mixed(fused._SplitRotate.apply(z, cos, sin)), x)
    _close(first, _penalty(lambda z: _mixed(_general(z, cos, sin)), x))


@pytest.mark.gpu
def test_on_the_gpu():
    x, t = _loss_case("cuda")
    _close(_penalty(lambda z: fused.token_cross_entropy(z, t), x), _penalty(lambda z: F.cross_entropy(z.float(), t), x))
    x, cos, sin = _rope_case("cuda")
    assert fused.split_rotate(x, cos, sin) is not None
    _close(_penalty(lambda z: _mixed(fused.split_rotate(z, cos, sin)), x), _penalty(lambda z: _mixed(_general(z, cos, sin)), x))
