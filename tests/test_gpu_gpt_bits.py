"""The GPT's training steps with the fused rotary embedding and loss have the bits of the operations they replace."""

import pytest
import torch
import torch.nn.functional as F
from torch.nn.attention import SDPBackend, sdpa_kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seq,batch", [(64, 1), (200, 3)])
def test_two_steps_have_the_bits_of_the_general_path(seq, batch, monkeypatch):
    """Losses, gradients and weights after two AdamW steps.  (The math attention: the flash backward adds dq in no fixed order,
    and from the second step on one flipped bit can send a token near a routing tie to another expert.)"""
    from ep_balance_b200.models import gpt_moe
    from ep_balance_b200.utils.optim import FusedAdamW

    def train():
        torch.manual_seed(0)
        cfg = gpt_moe.GPTMoEConfig(vocab=1024, layers=2, hidden=512, heads=4, ffn=256, experts=8, top_k=2, seq_len=seq,
                                   micro_batch=batch)
        model = gpt_moe.GPTMoE(cfg, torch.device("cuda", 0))
        dense = FusedAdamW(model.dense_parameters(), lr=1e-3)
        experts = FusedAdamW(list(model.expert_parameters()), lr=1e-3)
        ids = torch.randint(0, 1024, (batch, seq + 1), device="cuda")
        seen = {}
        for step in range(2):
            dense.zero_grad(set_to_none=True)
            loss = model(ids[:, :-1], ids[:, 1:])
            loss.backward()
            seen[f"loss {step}"] = loss.detach()
            for name, p in model.named_parameters():
                seen[f"{name} {step} grad"] = p.grad.clone()
            dense.step()
            experts.step()
        for name, p in model.named_parameters():
            seen[name] = p.detach().clone()
        model.check_status()
        return seen

    native, rotated = gpt_moe.split_rotate, []
    monkeypatch.setattr(gpt_moe, "split_rotate", lambda *a: rotated.append(native(*a)) or rotated[-1])
    with sdpa_kernel(SDPBackend.MATH):
        fused = train()
        assert len(rotated) == 4 and all(parts is not None for parts in rotated)
        monkeypatch.setattr(gpt_moe, "split_rotate", lambda *a: None)
        monkeypatch.setattr(gpt_moe, "token_cross_entropy", lambda z, t: F.cross_entropy(z.float(), t))
        general = train()
    assert [k for k in fused if not torch.equal(fused[k], general[k])] == []
