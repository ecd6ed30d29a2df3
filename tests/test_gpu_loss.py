"""Token cross-entropy from bf16 logits vs float64."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


# one vector, fewer vectors than threads, a partial step, an exact one; the last vocabulary takes the general path
@pytest.mark.parametrize("rows,vocab", [(1, 8), (3, 1000), (65, 32000), (7, 32768), (4, 70000), (6, 1001)])
def test_loss_and_gradient(rows, vocab):
    from ep_balance_b200.ops.fused import token_cross_entropy

    torch.manual_seed(0)
    x = (torch.randn(rows, vocab, device="cuda") * 4).bfloat16().requires_grad_(True)
    t = torch.randint(0, vocab, (rows,), device="cuda")
    t[0] = vocab - 1
    if rows > 2:
        t[1] = -100
    loss = token_cross_entropy(x, t)
    (loss * 0.5).backward()
    assert torch.equal(loss, F.cross_entropy(x.float(), t))
    ref = x.detach().double().requires_grad_(True)
    (F.cross_entropy(ref, t) * 0.5).backward()
    err = (x.grad.double() - ref.grad).norm() / ref.grad.norm()
    assert float(err) < 4e-3                                  # one bf16 rounding per value (2^-9 at most)
    if rows > 2:
        assert not bool(x.grad[1].any())


def test_special_rows():
    """-inf logits are zero probability, NaN rows and a batch without a counted target give NaN, as the library loss does."""
    from ep_balance_b200.ops.fused import token_cross_entropy

    x = torch.randn(4, 64, device="cuda").bfloat16()
    x[0, 5:] = float("-inf")
    t = torch.tensor([2, 7, 9, 63], device="cuda")
    assert abs(float(token_cross_entropy(x, t) - F.cross_entropy(x.float(), t))) < 1e-5
    assert bool(token_cross_entropy(x, torch.full_like(t, -100)).isnan())
    x[3, 1] = float("nan")
    assert bool(token_cross_entropy(x, t).isnan())
    full = torch.full((4, 64), float("-inf"), device="cuda").bfloat16()
    assert bool(token_cross_entropy(full, t).isnan())


@pytest.mark.parametrize("rows,vocab", [(1, 8), (65, 1000), (4096, 32000)])
@pytest.mark.parametrize("spread", [0.9, 8.0])
def test_gradient_has_the_bits_of_the_operations_it_replaces(rows, vocab, spread):
    from ep_balance_b200.ops.fused import token_cross_entropy

    torch.manual_seed(1)
    x = (torch.randn(rows, vocab, device="cuda") * spread).bfloat16()
    t = torch.randint(0, vocab, (rows,), device="cuda")
    t[1::7] = -100
    grads = []
    for f in (token_cross_entropy, lambda z, y: F.cross_entropy(z.float(), y)):
        z = x.clone().requires_grad_(True)
        (f(z, t) * 0.3).backward()
        grads.append(z.grad)
    assert torch.equal(*grads)
