"""The single-rank plan kernel vs the host semantics of the solver and the host model of the routing tables."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,zero", [(1, False), (8, False), (33, True), (128, False), (300, True), (1500, False)])
def test_plan_equals_host_semantics(E, zero):
    from ep_balance_b200 import EPLBConfig, Loads, ProblemSpec, Topology, solve
    from ep_balance_b200.solver import solve_device_semantics

    g = torch.Generator().manual_seed(E)
    omega = torch.randint(0, 700, (1, E), generator=g)
    if zero:
        omega[0, ::3] = 0
    topo, cfg = Topology.from_nvlink_rdma(1, 1), EPLBConfig()
    spec = ProblemSpec.contiguous_main_placement(E, 1, 1 << 20, 4096, E + 2)
    got = solve(Loads(omega.cuda()), topo.to("cuda"), spec.to("cuda"), cfg)
    want = solve_device_semantics(Loads(omega), topo, spec, cfg)
    assert got.to("cpu").equals(want)


@pytest.mark.parametrize("tokens,experts,top_k", [(1, 8, 2), (300, 40, 3), (512, 8, 8)])
def test_layer_tables(tokens, experts, top_k):
    from ep_balance_b200.models.emulated import EmulatedCluster
    from ep_balance_b200.models.moe_layer import MoEConfig
    from ep_balance_b200.parallel.transport_model import sender_tables

    torch.manual_seed(0)
    cfg = MoEConfig(hidden=256, ffn=256, num_experts=experts, top_k=top_k, max_tokens=512)
    layer = EmulatedCluster(cfg, world=1).layers[0]
    with torch.no_grad():
        layer(torch.randn(tokens, 256, device="cuda").bfloat16())
    layer.check_status()
    plan = layer.last_plan().to("cpu")
    x, q = plan.x.to(torch.int64), plan.q.to(torch.int64)
    want = sender_tables(x, q, layer.spec.main_rank.cpu(), 0, 128 * cfg.gemm_ctas)
    for name in ("row_base", "send_off", "tiles_of"):
        assert torch.equal(layer.loc[name].cpu().to(torch.int64), want[name]), name
    loc = {k: layer.loc[k].cpu() for k in ("group_expert", "group_wslot", "group_off", "group_rows", "slot_of", "totals", "rank_load",
                                           "slot_used", "theta", "erl", "stuck")}
    E, n = experts, q[0, :, 0]
    assert torch.equal(loc["group_expert"], torch.arange(E, dtype=torch.int32)) and torch.equal(loc["group_wslot"], loc["group_expert"])
    assert torch.equal(loc["slot_of"][:, 0], loc["group_expert"]) and torch.equal(loc["group_rows"].long(), n)
    padded = (n + 255) // 256 * 256
    assert torch.equal(loc["group_off"].long(), torch.cat([torch.zeros(1, dtype=torch.int64), padded.cumsum(0)]))
    assert loc["totals"].tolist() == [int(padded.sum()), E]
    assert torch.equal(loc["erl"][:, 0].long(), n)
    assert int(loc["rank_load"]) == int(loc["theta"]) == tokens * top_k and int(loc["slot_used"]) == E and int(loc["stuck"]) == 1
