"""CTA-pair grouped GEMM with the weights on the M side and ragged token rows as columns vs a plain fp32 loop over groups."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

MODE = dict(fwd1=0, fwd2=1, dgrad1=3, plain=5)
# around the 32-column step, the halves of the pair, one and several tiles of 256 (cut evenly), an empty group
ROWS = [1, 31, 32, 33, 0, 64, 255, 256, 257, 288, 512, 513, 900]
SLOTS = len(ROWS)
ATOL = 2 ** -8  # bf16 results of fp32 sums: half an ulp each, and the sums differ in order only


def _table():
    off, acc = [], 0
    for r in ROWS:
        off.append(acc)
        acc += -(-r // 256) * 256
    return off + [acc], acc


def _run(mode, k, n, w_shape):
    from ep_balance_b200.ops.extension import load

    torch.manual_seed(k + n)
    off, T = _table()
    a = torch.randn(T, k, device="cuda").bfloat16()
    for g, r in enumerate(ROWS):
        a[off[g] + r:off[g + 1]] = float("nan")  # rows outside the groups: none may reach a result
    w = (torch.randn(SLOTS, *w_shape, device="cuda") / k ** 0.5).bfloat16()
    slots = torch.randperm(SLOTS).tolist()
    out0 = torch.full((T, 2 * n if mode == "fwd1" else n), 7.0, device="cuda").bfloat16()
    out1 = torch.full((T, n), 7.0, device="cuda").bfloat16() if mode == "fwd1" else None
    i32 = dict(dtype=torch.int32, device="cuda")
    status = torch.zeros(4, **i32)
    load().grouped_gemm(MODE[mode], a, w, out0, out1, torch.tensor(off, **i32), torch.tensor(ROWS, **i32), torch.tensor(slots, **i32),
                        torch.tensor([T, SLOTS], **i32), status, torch.cuda.get_device_properties(0).multi_processor_count, 2)
    torch.cuda.synchronize()
    assert status.tolist()[0] == 0, status.tolist()
    return off, a, w, slots, out0, out1


def _close(got, want):
    torch.testing.assert_close(got.float(), want, rtol=ATOL, atol=ATOL)


# output columns that end inside a CTA's 128 or a 256-wide tile; reductions of an odd number of k-blocks and of a partial one;
# 96 columns are no multiple of 64 and take the single-CTA kernel
@pytest.mark.parametrize("mode,k,n", [("plain", 64, 32), ("plain", 200, 320), ("fwd2", 448, 576), ("dgrad1", 64, 64), ("dgrad1", 320, 448),
                                      ("dgrad1", 200, 384), ("dgrad1", 128, 96)])
def test_rows_at_tile_edges(mode, k, n):
    off, a, w, slots, out, _ = _run(mode, k, n, (k, n) if mode == "dgrad1" else (n, k))
    for g, r in enumerate(ROWS):
        wg = w[slots[g]].float()
        _close(out[off[g]:off[g] + r], a[off[g]:off[g] + r].float() @ (wg if mode == "dgrad1" else wg.t()))
        assert bool((out[off[g] + r:off[g + 1]] == 7.0).all())  # rows past the group's end are never written


@pytest.mark.parametrize("k,n", [(64, 128), (320, 384)])
def test_swiglu_and_zeroed_padding(k, n):
    off, a, w, slots, h, act = _run("fwd1", k, n, (2 * n, k))
    for g, r in enumerate(ROWS):
        sl = slice(off[g], off[g] + r)
        _close(h[sl], a[sl].float() @ w[slots[g]].float().t())
        gate, up = h[sl].float().chunk(2, dim=-1)
        _close(act[sl], F.silu(gate) * up)
        assert not bool(h[off[g] + r:off[g + 1]].any()) and not bool(act[off[g] + r:off[g + 1]].any())
