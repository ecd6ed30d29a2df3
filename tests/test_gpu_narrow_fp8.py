"""fp8 forward of few rows per expert (weights on the M side, activation in the first GEMM's epilogue) vs the wide kernels."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# one row; partial and full boxes of 32; several token tiles of one expert (skew); odd numbers of 128-feature blocks and
# k-groups that end early; the last batch below the rule (192 rows per expert) and the first past it
@pytest.mark.parametrize("H,F,E,K,N,skew", [(256, 128, 8, 2, 1, 0.0), (384, 640, 8, 2, 33, 2.0), (1280, 384, 16, 4, 300, 3.0),
                                            (512, 256, 8, 2, 767, 1.0), (512, 256, 8, 2, 768, 1.0)])
@pytest.mark.parametrize("ctas", [1, 2])
def test_matches_the_wide_kernels(H, F, E, K, N, skew, ctas):
    from ep_balance_b200.models.emulated import EmulatedCluster
    from ep_balance_b200.models.moe_layer import MoEConfig

    torch.manual_seed(0)
    cfg = MoEConfig(hidden=H, ffn=F, num_experts=E, top_k=K, max_tokens=768, fp8_inference=True, gemm_ctas=ctas)
    cl = EmulatedCluster(cfg, world=1)
    layer = cl.layers[0]
    layer.router_bias = torch.linspace(0, skew, E, device="cuda")
    layer.quantize_weights()
    x = torch.randn(N, H, device="cuda").bfloat16()
    (want,), _ = cl.forward_fp8([x])                     # piecewise: wide GEMMs, activation as a pass of its own
    for t in (layer._fp8_local["actq"], layer._fp8_local["sfact"]):
        t.fill_(0xFF)                                    # NaN bytes: rows and scales that nobody writes must not matter
    layer.rt.trace_launches(True)
    with torch.no_grad():
        got = layer(x)
    log = layer.rt.launch_log()
    layer.rt.trace_launches(False)
    layer.check_status()
    assert any("narrow" in n for n in log) == (N * K < 192 * E), log
    assert ("swiglu_quantize" in log) == (ctas == 1 and N * K >= 192 * E), log  # every other path finishes it in the first GEMM
    # same quantised operands; fp32 sums of K products in another order can move a pre-activation's bf16 rounding
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 1e-2
