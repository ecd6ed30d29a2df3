"""Fused inference router vs the PyTorch formulation in float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("N,H,E,K", [(1, 64, 8, 1), (37, 320, 40, 5), (1531, 512, 64, 8), (5, 128, 1024, 32)])
def test_split_logits_against_float64(mode, N, H, E, K):
    from ep_balance_b200.models.dsv3 import group_limited_topk
    from ep_balance_b200.ops.extension import load

    torch.manual_seed(0)
    G, keep, scale = (4, 3, 2.5) if mode == 2 else (1, 1, 1.0)
    x = torch.randn(N, H, device="cuda").bfloat16()
    w = torch.randn(E, H, device="cuda") * 0.05
    bias = 0.3 * torch.randn(E, device="cuda")
    stacked = torch.empty(3 * E, H, dtype=torch.bfloat16, device="cuda")
    load().router_split(w, stacked)
    assert float((stacked.double().view(3, E, H).sum(0) - w).norm() / w.norm()) < 2e-7  # 24 bits
    idx, prob = torch.empty((N, K), dtype=torch.int64, device="cuda"), torch.empty((N, K), device="cuda")
    load().router_topk(torch.mm(x, stacked.t(), out_dtype=torch.float32), bias, mode, G, keep, scale, idx, prob, 3)
    logits = x.double() @ w.double().t() + bias
    if mode == 2:
        ridx, _ = group_limited_topk(logits.float(), G, keep, K)
        top = torch.sigmoid(logits).gather(1, ridx)
        want = top / top.sum(-1, keepdim=True) * scale
    else:
        val, ridx = torch.topk(logits, K, dim=-1)
        want = torch.softmax(val, -1) if mode == 0 else torch.sigmoid(val)
    rows = (idx == ridx).all(1)           # a near tie may be ordered the other way in fp32
    assert float(rows.float().mean()) > 0.99
    assert float((prob - want)[rows].norm() / want[rows].norm()) < 4e-6   # fp32 logits of ~2, exponentiated


def test_masked_equal_and_nan_logits():
    from ep_balance_b200.ops.extension import load

    x = torch.randn(6, 70, device="cuda")
    x[0, 3:] = float("-inf")              # fewer candidates than K: distinct experts, weight 0
    x[1] = torch.finfo(torch.float32).min
    x[2] = 0.25
    x[3, 11] = float("nan")
    x[4, 11] = float("inf")
    idx, prob = torch.empty((6, 8), dtype=torch.int64, device="cuda"), torch.empty((6, 8), device="cuda")
    load().router_topk(x, None, 0, 1, 1, 1.0, idx, prob)
    assert all(len(set(r)) == 8 and 0 <= min(r) and max(r) < 70 for r in idx.tolist())
    want = torch.softmax(torch.topk(x, 8, dim=-1).values, -1)
    for r in (0, 1, 2, 5):
        assert torch.allclose(prob[r], want[r], atol=1e-6)
    assert bool(prob[3].isnan().all()) and bool(prob[4].isnan().all())
    assert idx[2].tolist() == list(range(8)) and int(idx[3, 0]) == 11


def test_a_nan_logit_spoils_its_own_sigmoid_weight_only():
    from ep_balance_b200.ops.extension import load

    x = torch.randn(3, 40, device="cuda")
    x[0, 33] = float("nan")
    x[1, 2] = float("inf")
    idx, prob = torch.empty((3, 4), dtype=torch.int64, device="cuda"), torch.empty((3, 4), device="cuda")
    load().router_topk(x, None, 1, 1, 1, 1.0, idx, prob)
    val, ridx = torch.topk(x, 4, dim=-1)
    assert torch.equal(idx, ridx)
    assert torch.allclose(prob, torch.sigmoid(val), atol=1e-6, equal_nan=True) and int(prob.isnan().sum()) == 1


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (64, 2048), (1531, 64), (8192, 160)])
def test_native_split_has_the_bits_of_the_operations(rows, cols):
    """Three bf16 terms of an fp32 matrix and of its transpose: tile edges of the transposing kernel, subnormals, infinities."""
    from ep_balance_b200.models.moe_layer import _split3

    torch.manual_seed(rows)
    w = torch.randn(rows, cols, device="cuda") * torch.logspace(-38, 30, cols, device="cuda")
    w[0, 0] = float("inf")
    w[-1, -1] = 1e-41
    for transposed in (False, True):
        with torch.no_grad():
            native = _split3(w, transposed)
        plain = _split3(w.clone().requires_grad_(True), transposed).detach()  # recorded: the operations themselves
        same = (native.view(torch.int16) == plain.view(torch.int16)) | (native.isnan() & plain.isnan())
        assert native.shape == plain.shape and bool(same.all())
