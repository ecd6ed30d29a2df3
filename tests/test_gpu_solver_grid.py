"""Plans whose quotas do not fit in shared memory: the whole grid routes, moves read the quotas from global memory."""

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
