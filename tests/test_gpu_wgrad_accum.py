"""fp32 accumulation of weight gradients in the Wgrad epilogue: sums of unrounded fp32 products, in place, where the tiles are
partial in either direction."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# 320 columns end inside a 256-wide tile and 320 rows inside a 256-row one; 1408 and 384 likewise, 576 rows inside the second CTA's half
@pytest.mark.parametrize("H,Fd", [(320, 384), (256, 1408), (576, 128)])
@pytest.mark.parametrize("ctas", [1, 2])
def test_accumulators_receive_the_unrounded_products(H, Fd, ctas):
    from ep_balance_b200.models.emulated import EmulatedCluster
    from ep_balance_b200.models.moe_layer import MoEConfig

    torch.manual_seed(0)
    E, N = 8, 300
    cl = EmulatedCluster(MoEConfig(hidden=H, ffn=Fd, num_experts=E, top_k=2, max_tokens=512, gemm_ctas=ctas,
                                   grad_accum_dtype=torch.float32), world=1)
    layer = cl.layers[0]
    bias = torch.linspace(0, 0.5, E, device="cuda")
    bias[3], bias[E - 1] = -30.0, 1.0  # an expert without rows, between others: what runs over a slot's end lands in the next
    layer.router_bias = bias
    start = [torch.randn_like(layer._acc_gw1), torch.randn_like(layer._acc_gw2)]
    layer._acc_gw1.copy_(start[0])
    layer._acc_gw2.copy_(start[1])
    want = [s.double() for s in start]
    for _ in range(2):
        x = torch.randn(N, H, device="cuda").bfloat16().requires_grad_(True)
        layer(x).backward(torch.randn(N, H, device="cuda").bfloat16())
        layer.check_status()
        # the operands as the GEMMs read them
        tokens, dy = cl.heap.tensor("xbuf", 0), cl.heap.tensor("dybuf", 0)
        dh, act = layer.loc["hbuf"], layer.loc["act"]
        rows = layer.loc["group_rows"].tolist()
        assert 0 in rows and sum(rows) == 2 * N
        for off, n, slot in zip(layer.loc["group_off"].tolist(), rows, layer.loc["group_wslot"].tolist()):
            sl = slice(off, off + n)
            want[0][slot] += dh[sl].double().t() @ tokens[sl].double()
            want[1][slot] += dy[sl].double().t() @ act[sl].double()
    for got, w, s in zip((layer.w1.main_grad, layer.w2.main_grad), want, start):
        added, empty = w - s.double(), 0
        for slot in range(E):
            if not bool(added[slot].any()):  # no rows: untouched
                assert torch.equal(got[slot], s[slot])
                empty += 1
                continue
            # fp32 sums of at most 600 products, added twice to values of the size of 1 (2^-24 each); a rounding to bf16 costs 1e-3
            err = float((got[slot].double() - w[slot]).norm())
            assert err < 2e-5 * float(added[slot].norm()) + 2 ** -23 * float(w[slot].norm())
        assert 0 < empty < E - 1
    assert layer.w1.grad is None and layer.w2.grad is None
