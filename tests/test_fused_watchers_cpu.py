"""Whoever has to see the operations (tracers, dispatch and function modes, subclasses, transforms) gets the PyTorch path of the
fused dense pieces, never a kernel launch."""

import pytest
import torch
import torch.nn.functional as F
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.fx.experimental.proxy_tensor import make_fx
from torch.overrides import TorchFunctionMode
from torch.utils.flop_counter import FlopCounterMode

from ep_balance_b200.models.dsv3 import SharedExpert
from ep_balance_b200.ops import fused

B, S, HEADS, DIM, VOCAB = 2, 4, 2, 16, 24


@pytest.fixture
def pretend_cuda(monkeypatch):
    """CPU tensors pass the device checks, and a kernel that is reached all the same fails the test."""
    def reached():
        raise AssertionError("a native kernel was reached")
    monkeypatch.setattr(fused, "load", reached)
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda self: True))


def _bf16(*shape, device="cpu"):
    return torch.randn(*shape, device=device).bfloat16()


def _all_pieces(device="cpu"):
    """One call of every public function, on tensors its kernel covers."""
    x, t = _bf16(6, VOCAB, device=device), torch.zeros(6, dtype=torch.int64, device=device)
    qkv, tab = _bf16(B, S, 3, HEADS, DIM, device=device), _bf16(S, DIM // 2, device=device)
    a = _bf16(4, 32, device=device)
    with torch.no_grad():
        out = [fused.swiglu(a), fused.add3(a, a, a)]
    rotated = fused.split_rotate(qkv, tab, tab)
    return out + [fused.token_cross_entropy(x, t)], rotated


class _Watch(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Sub(torch.Tensor):
    pass


def test_plain_calls_reach_the_kernels(pretend_cuda):
    a = _bf16(4, 32)
    for context in (torch.no_grad(), torch.inference_mode()):
        with context, pytest.raises(AssertionError):
            fused.swiglu(a)
    with torch.no_grad(), torch.device("cpu"), pytest.raises(AssertionError):  # a function mode that only sets defaults
        fused.add3(a, a, a)
    with pytest.raises(AssertionError):
        fused.split_rotate(_bf16(B, S, 3, HEADS, DIM), _bf16(S, DIM // 2), _bf16(S, DIM // 2))


def test_fake_tensors_flop_counters_and_function_modes(pretend_cuda):
    for watcher in (FakeTensorMode(), FlopCounterMode(display=False), _Watch()):
        with watcher:
            out, rotated = _all_pieces("cuda" if isinstance(watcher, FakeTensorMode) else "cpu")
        assert rotated is None and [tuple(o.shape) for o in out] == [(4, 16), (4, 32), ()]


def test_subclasses_and_transforms(pretend_cuda):
    a = _bf16(3, 4, 32)
    with torch.no_grad():
        assert fused.swiglu(a[0].as_subclass(_Sub)).shape == (4, 16)
        assert torch.equal(torch.vmap(fused.swiglu)(a), F.silu(a[..., :16]) * a[..., 16:])
    _, tangent = torch.func.jvp(lambda z: fused.token_cross_entropy(z, torch.zeros(4, dtype=torch.int64)), (a[0],), (a[1],))
    assert bool(tangent.isfinite())
    g = torch.func.grad(lambda z: fused.token_cross_entropy(z, torch.zeros(4, dtype=torch.int64)))(a[0])
    assert g.shape == a[0].shape


def _expert():
    torch.manual_seed(0)
    return SharedExpert(16, 16).bfloat16()


@pytest.mark.parametrize("tracer", ["jit.trace", "jit.script", "make_fx", "symbolic_trace", "compile", "export"])
def test_traced_shared_expert_computes(pretend_cuda, monkeypatch, tracer):
    m, x, y = _expert(), _bf16(4, 16), _bf16(4, 16)
    with torch.no_grad():
        if tracer == "jit.trace":
            f = torch.jit.trace(m, x, check_trace=False)  # (the check runs the module itself again)
        elif tracer == "jit.script":
            f = torch.jit.script(m)
        elif tracer == "make_fx":
            f = make_fx(m)(x)
        elif tracer == "symbolic_trace":
            f = torch.fx.symbolic_trace(m)
        elif tracer == "compile":
            f = torch.compile(m, backend="eager", fullgraph=True)
        else:
            f = torch.export.export(m, (x,)).module()
        gate, up = F.linear(y, m.up.weight).chunk(2, dim=-1)
        assert torch.equal(f(y), F.linear(F.silu(gate) * up, m.down.weight))


def test_inference_router(pretend_cuda, monkeypatch):
    """Forward-mode AD and modes get _RouterLinear, which refuses what it has no rule for; a plain call splits natively."""
    from types import SimpleNamespace

    from torch.autograd import forward_ad

    from ep_balance_b200.models import moe_layer

    class Reached(Exception):
        pass

    def general(*args):
        raise Reached
    monkeypatch.setattr(moe_layer, "load", fused.load)
    monkeypatch.setattr(moe_layer._RouterLinear, "apply", general)
    layer = SimpleNamespace(router=torch.nn.Parameter(torch.randn(8, 16)), _fused_routing=lambda: True)
    x = _bf16(4, 16)
    with torch.no_grad():
        with pytest.raises(AssertionError):
            moe_layer.FusedMoE.route_tokens(layer, x)
        with FlopCounterMode(display=False), pytest.raises(Reached):
            moe_layer.FusedMoE.route_tokens(layer, x)
        with forward_ad.dual_level(), pytest.raises(Reached):
            moe_layer.FusedMoE.route_tokens(layer, forward_ad.make_dual(x, x))
        with pytest.raises(Reached):
            torch.vmap(lambda z: moe_layer.FusedMoE.route_tokens(layer, z)[1])(_bf16(3, 4, 16))
