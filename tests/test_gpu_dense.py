"""One-pass SwiGLU and three-term sum of an inference forward: the bits of the operations they replace."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,f", [(1, 8), (7, 24), (300, 2048), (0, 16), (5, 12)])
def test_same_bits(rows, f):
    from ep_balance_b200.ops.fused import add3, swiglu

    torch.manual_seed(0)
    x = (4 * torch.randn(rows, 2 * f, device="cuda")).bfloat16()
    if rows > 1:
        x[0, 0], x[0, 1], x[1, 2] = float("nan"), float("inf"), float("-inf")
    gate, up = x.chunk(2, dim=-1)
    a, b, c = (torch.randn(rows, f, device="cuda").bfloat16() for _ in range(3))
    with torch.no_grad():
        got = swiglu(x), add3(a, b, c)
    for g, w in zip(got, (F.silu(gate) * up, a + b + c)):
        assert g.shape == w.shape and torch.equal(g.isnan(), w.isnan()) and torch.equal(g.nan_to_num(1.0), w.nan_to_num(1.0))


def test_autograd_and_other_layouts_keep_the_general_path():
    from ep_balance_b200.ops.fused import add3, swiglu

    x = torch.randn(4, 64, device="cuda").bfloat16().requires_grad_(True)
    add3(swiglu(x), x[:, :32], x[:, 32:]).sum().backward()
    assert x.grad is not None
    with torch.no_grad():
        y = x.detach().t()
        assert torch.equal(swiglu(y), F.silu(y.chunk(2, -1)[0]) * y.chunk(2, -1)[1])
        assert torch.equal(add3(y, y, y), y + y + y)
        assert torch.equal(add3(y, y[:1], y), y + y[:1] + y)
        assert add3(x, x.float(), x).dtype == torch.float32
