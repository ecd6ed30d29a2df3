"""Plans whose quotas do not fit in shared memory, or have a floor: routing has a launch of its own, moves read the quotas from
global memory."""

import pytest
import torch

pytestmark = pytest.mark.gpu


# one domain on a grid of many CTAs; ranks that end inside a warp, at its edge, past it and at 64; a quota floor
@pytest.mark.parametrize("domains,per_domain,per_rank,extra,u_min", [(1, 64, 1, 2, 1), (3, 11, 4, 1, 1), (2, 16, 12, 2, 1), (8, 8, 4, 2, 1),
                                                                     (2, 20, 5, 3, 1), (8, 8, 4, 2, 3), (1, 33, 8, 1, 2)])
@pytest.mark.parametrize("skew", [1.1, 1.5])
def test_plan_equals_host_semantics(domains, per_domain, per_rank, extra, u_min, skew):
    from ep_balance_b200 import EPLBConfig, ProblemSpec, Topology, solve
    from ep_balance_b200.core.loads import Loads
    from ep_balance_b200.solver import solve_device_semantics
    from ep_balance_b200.utils.workload import make_loads

    R = domains * per_domain
    E = R * per_rank
    topo = Topology.from_nvlink_rdma(domains, per_domain)
    spec = ProblemSpec.contiguous_main_placement(E, R, 3 * 2048 * 1408 * 2, 2 * 2048, per_rank + extra)
    cfg = EPLBConfig(u_min=u_min)
    om = make_loads(R, E, 2048, 6, skew, 0.25, 1).omega
    loads = Loads(torch.where((om > 0) & (om < u_min), torch.full_like(om, u_min), om).cuda())
    for _ in range(2):  # the second solve starts from a used workspace
        got = solve(loads, topo.to("cuda:0"), spec.to("cuda:0"), cfg, validate=False)
    want = solve_device_semantics(Loads(loads.omega.cpu()), topo, spec, cfg)
    assert got.to("cpu").equals(want)


def _problem(domains, per_domain, per_rank, u_min=1):
    from ep_balance_b200 import EPLBConfig, ProblemSpec, Topology
    from ep_balance_b200.core.loads import Loads
    from ep_balance_b200.utils.workload import make_loads

    R = domains * per_domain
    E = R * per_rank
    om = make_loads(R, E, 2048, 6, 1.3, 0.25, 1).omega
    om = torch.where((om > 0) & (om < u_min), torch.full_like(om, u_min), om)
    return (Topology.from_nvlink_rdma(domains, per_domain), ProblemSpec.contiguous_main_placement(E, R, 3 * 2048 * 1408 * 2, 4096, per_rank + 2),
            EPLBConfig(u_min=u_min), Loads(om.to(torch.int32)))


# on both sides of the size from which routing has a launch of its own (1024 pairs), rows of q of one to 64 entries
@pytest.mark.parametrize("domains,per_domain,per_rank", [(1, 2, 3), (2, 4, 8), (3, 5, 4), (2, 8, 4), (1, 13, 13), (5, 9, 2)])
def test_quota_floor(domains, per_domain, per_rank):
    from ep_balance_b200 import solve
    from ep_balance_b200.core.loads import Loads
    from ep_balance_b200.solver import solve_device_semantics

    topo, spec, cfg, loads = _problem(domains, per_domain, per_rank, u_min=3)
    for _ in range(2):
        got = solve(Loads(loads.omega.cuda()), topo.to("cuda:0"), spec.to("cuda:0"), cfg, validate=False)
    assert got.to("cpu").equals(solve_device_semantics(loads, topo, spec, cfg))


def test_unfit_inputs_leave_the_workspace_idle():
    from ep_balance_b200 import solve
    from ep_balance_b200.core.loads import Loads
    from ep_balance_b200.ops import solver_op
    from ep_balance_b200.solver import solve_device_semantics

    topo, spec, cfg, loads = _problem(8, 8, 4)
    dev = torch.device("cuda:0")
    omega, topo_d, spec_d = Loads(loads.omega.cuda()), topo.to("cuda:0"), spec.to("cuda:0")
    solve(omega, topo_d, spec_d, cfg, validate=False)
    ws = solver_op.workspace(64, 256, dev)
    dom = solver_op._static_inputs(topo_d, spec_d, dev)[0]
    good = dom.clone()
    dom[17] = 99
    solve(omega, topo_d, spec_d, cfg, validate=False)
    assert ws.status.tolist()[0] != 0 and ws.sync.tolist() == [0, 0]
    dom.copy_(good)
    ws.status.zero_()
    got = solve(omega, topo_d, spec_d, cfg, validate=False)
    assert ws.status.tolist()[0] == 0 and ws.sync.tolist() == [0, 0]
    assert got.to("cpu").equals(solve_device_semantics(loads, topo, spec, cfg))


def test_a_large_plan_runs_beside_a_gemm_that_leaves_it_a_few_sms():
    from ep_balance_b200 import solve
    from ep_balance_b200.core.loads import Loads
    from ep_balance_b200.ops.extension import load

    topo, spec, cfg, loads = _problem(8, 8, 4)
    topo, spec, loads = topo.to("cuda:0"), spec.to("cuda:0"), Loads(loads.omega.cuda())
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T, K, N = 262144, 4096, 16384  # 35 TFLOP: at least 15 ms, a plan and its launches take about one
    a = torch.zeros(T, K, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(1, N, K, dtype=torch.bfloat16, device="cuda")
    out = torch.empty(T, N, dtype=torch.bfloat16, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    tables = [torch.tensor(v, **i32) for v in ([0, T], [T], [0], [T, 1])]
    status = torch.zeros(4, **i32)
    gemm = lambda: load().grouped_gemm(1, a, w, out, None, *tables, status, sms - 20, 2)  # noqa: E731
    gemm()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    gemm_done, plan_done = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    with torch.cuda.stream(side):
        for _ in range(3):  # (its outputs' memory is this stream's from here on: an allocation could wait for the device)
            solve(loads, topo, spec, cfg, validate=False)
    torch.cuda.synchronize()
    gemm()
    gemm_done.record()
    with torch.cuda.stream(side):
        solve(loads, topo, spec, cfg, validate=False)
        plan_done.record()
    torch.cuda.synchronize()
    assert plan_done.elapsed_time(gemm_done) > 0  # by the device's clock
    assert status.tolist()[0] == 0
