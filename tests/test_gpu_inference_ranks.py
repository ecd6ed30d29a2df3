"""Inference forwards of four emulated ranks with the kernels that a layer's own forward picks without autograd, vs the oracle:
replicas, rows from and to other ranks, no padding rows, and ranks on both sides of the rule for few rows per expert."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

WORLD, E, K = 4, 16, 2  # 4 owned experts + 2 replica slots a rank: the rules' lines are at 384 (bf16) and 576 (fp8) tokens


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12))


def _cluster(H, Fd, **kw):
    from ep_balance_b200.models.emulated import EmulatedCluster
    from ep_balance_b200.models.moe_layer import MoEConfig

    torch.manual_seed(0)
    cl = EmulatedCluster(MoEConfig(hidden=H, ffn=Fd, num_experts=E, top_k=K, max_tokens=700, extra_slots=2,
                                   capacity_factor=float(WORLD), **kw), world=WORLD)
    bias = torch.zeros(E, device="cuda")
    bias[:3], bias[5] = 3.0, -30.0  # three hot experts, one that nobody asks for
    for r, l in enumerate(cl.layers):
        l.router_bias = bias
        for t in (l.loc["act"], l.loc["hbuf"], cl.heap.tensor("xbuf", r), cl.heap.tensor("ybuf", r)):
            t.fill_(float("nan"))  # what nobody writes must not matter
    return cl


def _run(cl, tokens, call):
    for l in cl.layers:
        l.rt.trace_launches(True)
    outs, routing = call(tokens)
    torch.cuda.synchronize()
    cl.status.check_now()
    assert int(cl.layers[0].last_plan().x.sum()) > E  # replicas exist
    assert cl.heap.damaged_guards() == []
    return outs, routing, [l.rt.launch_log() for l in cl.layers]


@pytest.mark.parametrize("ctas", [1, 2])
@pytest.mark.parametrize("counts", [(1, 17, 130, 384), (384, 385, 3, 700), (700, 600, 500, 400)])
def test_bf16(counts, ctas):
    from ep_balance_b200.models.reference_moe import moe_reference

    cl = _cluster(320, 384, gemm_ctas=ctas)
    tokens = [torch.randn(n, 320, device="cuda").bfloat16() for n in counts]
    outs, routing, logs = _run(cl, tokens, cl.infer)
    assert [sum("narrow" in x for x in log) for log in logs] == [2 * (n <= 384) for n in counts]
    w1, w2 = cl.full_weights()
    for x, out, (idx, prob) in zip(tokens, outs, routing):
        assert _rel(out, moe_reference(x.float(), idx, prob, w1.float(), w2.float())) < 2e-2


def _quantised(x):
    """fp32 [rows, n] -> the values that e4m3 with one power-of-two scale per 1 x 128 block represents."""
    b = x.view(x.shape[0], -1, 128)
    e = torch.ceil(torch.log2(b.abs().amax(-1, keepdim=True).double() / 448)).clamp(-126, 126).float()
    return ((b * torch.exp2(-e)).to(torch.float8_e4m3fn).float() * torch.exp2(e)).view_as(x)


def _fp8_oracle(x, idx, prob, w1, w2):
    """The layer's math in fp32 on the quantised operands, with the pre-activations and the expert rows rounded to bf16."""
    out = torch.zeros_like(x, dtype=torch.float32)
    xq = _quantised(x.float())
    for e in torch.unique(idx).tolist():
        t, k = (idx == e).nonzero(as_tuple=True)
        gate, up = (xq[t] @ w1[e].t()).bfloat16().float().chunk(2, dim=-1)
        y = (_quantised(F.silu(gate) * up) @ w2[e].t()).bfloat16().float()
        out.index_add_(0, t, prob[t, k, None] * y)
    return out


@pytest.mark.parametrize("H,Fd", [(384, 640), (256, 1408)])
@pytest.mark.parametrize("ctas", [1, 2])
@pytest.mark.parametrize("counts", [(1, 33, 257, 575), (575, 576, 5, 700), (700, 690, 680, 670)])
def test_fp8(counts, ctas, H, Fd):
    from ep_balance_b200.ops.fp8 import dequantize_weights, quantize_weights

    cl = _cluster(H, Fd, gemm_ctas=ctas, fp8_inference=True)
    for l in cl.layers:
        l.quantize_weights()
        for name in ("actq", "sfact"):
            l._fp8_local[name].fill_(0xFF)
    tokens = [torch.randn(n, H, device="cuda").bfloat16() for n in counts]
    outs, routing, logs = _run(cl, tokens, lambda t: cl.forward_fp8(t, general=False))
    assert [sum("narrow" in x for x in log) for log in logs] == [2 * (n < 576) for n in counts]
    assert ["swiglu_quantize" in log for log in logs] == [ctas == 1 and n >= 576 for n in counts]
    w1, w2 = (dequantize_weights(*quantize_weights(w.contiguous())) for w in cl.full_weights())
    for x, out, (idx, prob) in zip(tokens, outs, routing):
        # bf16 roundings of the expert rows and of the sum (2^-9 at most each), and a pre-activation that rounds the other
        # way in another order of summation can move an activation to its e4m3 neighbour
        assert _rel(out, _fp8_oracle(x, idx, prob, w1, w2)) < 8e-3
