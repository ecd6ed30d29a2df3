"""Packed projection -> rotated q, k and v (and the gradient) vs the elementwise formulation in float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,heads,dim", [(1, 1, 1, 16), (2, 37, 3, 48), (1, 257, 16, 128)])
@pytest.mark.parametrize("transposed_grad", [False, True])
def test_split_rotate(B, S, heads, dim, transposed_grad):
    from ep_balance_b200.models.gpt_moe import apply_rope, rope_tables
    from ep_balance_b200.ops.fused import split_rotate

    torch.manual_seed(0)
    cos, sin = rope_tables(S + 5, dim, 10000.0, "cuda", torch.bfloat16)
    cos, sin = cos[:S], sin[:S]
    x = torch.randn(B, S, 3, heads, dim, device="cuda").bfloat16().requires_grad_(True)
    parts = split_rotate(x, cos, sin)
    assert parts is not None
    grads = [torch.randn(B, S, heads, dim, device="cuda").bfloat16().transpose(1, 2) for _ in range(3)]
    if not transposed_grad:
        grads = [g.contiguous() for g in grads]
    torch.autograd.backward(parts, grads)
    ref = x.detach().double().requires_grad_(True)
    q, k, v = ref.permute(2, 0, 3, 1, 4)
    want = apply_rope(q, cos.double(), sin.double()), apply_rope(k, cos.double(), sin.double()), v
    torch.autograd.backward(want, [g.double() for g in grads])
    for a, b in zip((*parts, x.grad), (*want, ref.grad)):
        assert float((a.double() - b).norm() / b.norm()) < 8e-3  # two bf16 roundings per value (2^-9 at most each)
    q, k, v = x.detach().permute(2, 0, 3, 1, 4)
    for a, b in zip(parts, (apply_rope(q, cos, sin), apply_rope(k, cos, sin), v)):  # the general path, bit for bit
        assert torch.equal(a, b)


def test_other_layouts_take_the_general_path():
    from ep_balance_b200.ops.fused import split_rotate

    cos = torch.ones(4, 8, device="cuda").bfloat16()
    x = torch.randn(1, 4, 3, 2, 16, device="cuda").bfloat16()
    assert split_rotate(x, cos, cos) is not None
    assert split_rotate(x.transpose(0, 1).contiguous().transpose(0, 1)[:, :, :, :, ::1].expand(2, -1, -1, -1, -1), cos, cos) is None
    assert split_rotate(x.float(), cos, cos) is None
    assert split_rotate(x, cos.float(), cos) is None
    assert split_rotate(x[..., :8], cos[:, :4], cos[:, :4]) is None


@pytest.mark.parametrize("B,S,heads,dim", [(1, 1, 1, 16), (3, 37, 3, 48), (2, 2048, 16, 128)])
def test_gradient_has_the_bits_of_the_operations_it_replaces(B, S, heads, dim):
    """Gradients laid out as attention's backward hands them over: q and k per head, v per position."""
    from ep_balance_b200.models.gpt_moe import apply_rope, rope_tables
    from ep_balance_b200.ops.fused import split_rotate

    torch.manual_seed(1)
    cos, sin = rope_tables(S, dim, 10000.0, "cuda", torch.bfloat16)
    x = torch.randn(B, S, 3, heads, dim, device="cuda").bfloat16()
    dq, dk = (torch.randn(B, heads, S, dim, device="cuda").bfloat16() for _ in range(2))
    dv = torch.randn(B, S, heads, dim, device="cuda").bfloat16().transpose(1, 2)
    grads, strides = [], []
    for general in (False, True):
        z = x.clone().requires_grad_(True)
        if general:
            q, k, v = z.permute(2, 0, 3, 1, 4)
            parts = apply_rope(q, cos, sin), apply_rope(k, cos, sin), v
        else:
            parts = split_rotate(z, cos, sin)
        torch.autograd.backward(parts, [dq, dk, dv])
        grads.append(z.grad)
        strides.append([p.stride() for p in parts])
    assert torch.equal(*grads) and strides[0] == strides[1]  # (the strides choose attention's kernel)
