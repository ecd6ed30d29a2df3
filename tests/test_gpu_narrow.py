"""Grouped GEMM with the weights on the M side (few rows per expert) vs a plain fp32 loop over groups, and the layer's
inference forward, which selects it, vs the oracle."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

MODE = dict(fwd1=0, fwd2=1)
# one row, a partial and a full 16-column step, box and tile edges (32, 128), two and three token tiles, an empty group
ROWS = [1, 0, 16, 33, 128, 129, 300]
WSLOT = [3, 0, 6, 1, 2, 5, 4]


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12))


def _run(mode, a, w, out0, out1, tile=256):
    from ep_balance_b200.ops.extension import load

    off, acc = [], 0
    for r in ROWS:
        off.append(acc)
        acc += -(-r // tile) * tile
    off.append(acc)
    i32 = dict(dtype=torch.int32, device="cuda")
    status = torch.zeros(4, **i32)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    load().grouped_gemm(MODE[mode], a, w, out0, out1, torch.tensor(off, **i32), torch.tensor(ROWS, **i32),
                        torch.tensor(WSLOT, **i32), torch.tensor([acc, len(ROWS)], **i32), status, sms, 2, narrow=True)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0, status.tolist()
    return off


def _rows_total(tile=256):
    return sum(-(-r // tile) * tile for r in ROWS)


def _operand(T, K):
    """Rows outside the groups are NaN: none of them may reach a result."""
    a = torch.randn(T, K, device="cuda").bfloat16()
    off = 0
    for r in ROWS:
        end = off + -(-r // 256) * 256
        a[off + r:end] = float("nan")
        off = end
    return a


@pytest.mark.parametrize("N,K", [(64, 64), (256, 192), (320, 1408), (2048, 768)])
def test_plain_rows(N, K):
    torch.manual_seed(0)
    T = _rows_total()
    a = _operand(T, K)
    w = (torch.randn(7, N, K, device="cuda") * 0.05).bfloat16()
    out = torch.full((T, N), 7.0, device="cuda").bfloat16()
    off = _run("fwd2", a, w, out, None)
    for g, r in enumerate(ROWS):
        want = a[off[g]:off[g] + r].float() @ w[WSLOT[g]].float().t()
        if r:
            assert _rel(out[off[g]:off[g] + r], want) < 4e-3  # one bf16 rounding (2^-9 at most) of an fp32 sum
        assert bool((out[off[g] + r:off[g + 1]] == 7.0).all())


@pytest.mark.parametrize("Fd,K", [(128, 64), (384, 512)])
def test_swiglu(Fd, K):
    torch.manual_seed(1)
    T = _rows_total()
    a = _operand(T, K)
    w = (torch.randn(7, 2 * Fd, K, device="cuda") * 0.05).bfloat16()
    act = torch.full((T, Fd), 3.0, device="cuda").bfloat16()
    off = _run("fwd1", a, w, act[:0], act)  # (no buffer for the pre-activations)
    for g, r in enumerate(ROWS):
        sl = slice(off[g], off[g] + r)
        hh = a[sl].float() @ w[WSLOT[g]].float().t()
        if r:
            gate, up = hh.bfloat16().float().chunk(2, dim=-1)
            assert _rel(act[sl], F.silu(gate) * up) < 1e-2  # three bf16 roundings: gate, up, product
        assert bool((act[off[g] + r:off[g + 1]] == 3.0).all())


@pytest.mark.parametrize("tokens,experts,fused_comm", [(1, 8, True), (65, 16, True), (512, 8, True), (700, 8, True), (65, 16, False)])
def test_inference_forward_both_sides_of_the_rule(tokens, experts, fused_comm):
    """512 tokens x 2 = 128 rows per expert: the last batch on the narrow kernel; 700 are past it."""
    from ep_balance_b200.models.emulated import EmulatedCluster
    from ep_balance_b200.models.moe_layer import MoEConfig
    from ep_balance_b200.models.reference_moe import moe_reference

    torch.manual_seed(2)
    cfg = MoEConfig(hidden=320, ffn=384, num_experts=experts, top_k=2, max_tokens=700, fused_comm=fused_comm)
    cl = EmulatedCluster(cfg, world=1)
    layer = cl.layers[0]
    layer.router_bias = torch.linspace(0, 2.0, experts, device="cuda")
    x = torch.randn(tokens, 320, device="cuda").bfloat16()
    for t in (layer.loc["act"], layer.loc["hbuf"], cl.heap.tensor("xbuf", 0)):
        t.fill_(float("nan"))  # what an inference pass leaves unwritten must not matter
    layer.rt.trace_launches(True)
    with torch.no_grad():
        out = layer(x)
    log = layer.rt.launch_log()
    layer.rt.trace_launches(False)
    layer.check_status()
    assert any("narrow" in n for n in log) == (tokens * 2 <= 128 * experts), log
    idx, prob = layer.route_tokens(x)
    w1, w2 = cl.full_weights()
    assert _rel(out, moe_reference(x.float(), idx, prob.detach(), w1.float(), w2.float())) < 2e-2
    # a training pass after it is complete again (padding rows, pre-activations)
    tok = x.clone().requires_grad_(True)
    layer(tok).sum().backward()
    layer.check_status()
    for g in (tok.grad, layer.w1.grad, layer.w2.grad):
        assert torch.isfinite(g.float()).all()


@pytest.mark.parametrize("tokens", [65, 700])
def test_fused_trace_of_an_inference_forward(tokens, monkeypatch):
    """The profiling aid sees the transport and the GEMM on both sides of the rule."""
    from ep_balance_b200.models.emulated import EmulatedCluster
    from ep_balance_b200.models.moe_layer import MoEConfig

    monkeypatch.setenv("EPLB_TRACE_FUSED", "1")
    layer = EmulatedCluster(MoEConfig(hidden=320, ffn=384, num_experts=8, top_k=2, max_tokens=700), world=1).layers[0]
    layer.fused_trace_reset()
    with torch.no_grad():
        layer(torch.randn(tokens, 320, device="cuda").bfloat16())
    layer.check_status()
    trace = layer.fused_trace()
    assert 0 < trace["fwd_first_tile_us"] <= trace["fwd_mma_end_us"] < 1e5 and 0 < trace["fwd_transport_us"] < 1e5
    assert trace["fwd_warp_segments"] > 0
