"""The extension refuses tensors that have no memory, before anything is launched.  Runs on the CPU: no such call may reach a GPU."""

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from ep_balance_b200.ops.extension import load


@pytest.mark.skipif(torch.cuda.is_available(), reason="a call that should be refused is not made where a GPU could run it")
def test_fake_tensors_are_refused():
    ext = load()
    with FakeTensorMode():
        bf = lambda *s: torch.empty(s, dtype=torch.bfloat16, device="cuda")  # noqa: E731
        f32 = lambda *s: torch.empty(s, device="cuda")                       # noqa: E731
        i64 = lambda *s: torch.empty(s, dtype=torch.int64, device="cuda")    # noqa: E731
        a, q = bf(4, 32), bf(1, 2, 4, 16)
        for call in (lambda: ext.swiglu(a, bf(4, 16)), lambda: ext.add3(a, a, a, a), lambda: ext.router_split(f32(8, 16), bf(24, 16)),
                     lambda: ext.router_topk(f32(4, 8), None, 0, 1, 1, 1.0, i64(4, 2), f32(4, 2)),
                     lambda: ext.rope(bf(1, 4, 3, 2, 16), q, q, q, bf(4, 8), bf(4, 8), True),
                     lambda: ext.cross_entropy_backward(f32(4, 8), i64(4), f32(), f32(), bf(4, 8))):
            with pytest.raises(RuntimeError, match="no memory"):
                call()
