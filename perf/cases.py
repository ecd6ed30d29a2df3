"""The work a program built on this package gives it, as a list of timed cases.

Four families, each through its public entry points:

``plan``    ``solve`` for a load matrix that lives on the GPU: what every layer of every micro-batch pays.
``layer``   one ``FusedMoE`` layer: training steps (eager or replayed from a CUDA graph, with ``FusedAdamW``;
            one batch or several accumulated in fp32) and bf16 inference.
``stack``   the DeepSeek-V3-shaped block (hidden 7168, group-limited routing, shared expert): training in bf16,
            inference in bf16 and with block-scaled fp8 experts.
``gpt``     a training step of the GPT with MoE blocks.

Everything runs on one GPU.  Sizes are those of ``bench.py``, ``launch/recipes.py`` and the launchers' defaults, or
generic; token counts are also odd and ragged, and smaller than the ``max_tokens`` a program reserves.
"""

from __future__ import annotations

import math

import torch

from ep_balance_b200 import EPLBConfig, Loads, ProblemSpec, Topology, solve
from ep_balance_b200.launch.recipes import RECIPES
from ep_balance_b200.models.dsv3 import DSv3Config, DSv3Stack
from ep_balance_b200.models.gpt_moe import GPTMoE, GPTMoEConfig
from ep_balance_b200.models.moe_layer import FusedMoE, MoEConfig, heap_layout
from ep_balance_b200.parallel.symm import SymmetricHeap
from ep_balance_b200.utils.graphs import GraphedStep
from ep_balance_b200.utils.optim import FusedAdamW
from ep_balance_b200.utils.workload import make_loads

DEVICE = "cuda:0"
STACK = dict(hidden=7168, ffn=2048)  # the DeepSeek-V3 layer; 32 experts are one GPU's share of 256 over 8


def listed():
    return [
        # the plan of one layer on the bench's 8 ranks (2 domains of 4, 2 spare slots): latency, once per layer and step
        dict(name="plan_64e_8r", kind="plan", experts=64, domains=2, per_domain=4, extra=2, skew=1.2, top_k=6),
        # the same on eight nodes of eight GPUs with 256 experts
        dict(name="plan_256e_64r", kind="plan", experts=256, domains=8, per_domain=8, extra=2, skew=1.4, top_k=8),
        # a step of the bring-up recipe: tiny sizes, launched eagerly, so that the host and the launches count
        dict(name="layer_step_tiny", kind="layer", mode="step", graph=False, hidden=512, ffn=512, experts=8, top_k=2,
             tokens=200, max_tokens=512, micro=1, skew=0.3),
        # the bench's training step: forward, loss, backward, AdamW, replayed from a CUDA graph
        dict(name="layer_step_8192", kind="layer", mode="step", graph=True, hidden=2048, ffn=1408, experts=64, top_k=6,
             tokens=8192, max_tokens=8192, micro=1, skew=0.35),
        # two ragged micro-batches accumulated in fp32 before the optimizer, eager: the GPT recipe's layer in a pipeline
        dict(name="layer_accum_1531", kind="layer", mode="step", graph=False, hidden=2048, ffn=1024, experts=64, top_k=8,
             tokens=1531, max_tokens=2048, micro=2, skew=0.35),
        # bf16 inference of a small batch against many experts: bound by reading the weights
        dict(name="layer_infer_64", kind="layer", mode="infer", graph=False, hidden=2048, ffn=768, experts=128, top_k=8,
             tokens=64, max_tokens=4096, micro=1, skew=0.35),
        # bf16 prefill, ragged, 160 experts with few rows each: tile padding counts
        dict(name="layer_infer_3001", kind="layer", mode="infer", graph=False, hidden=5120, ffn=1536, experts=160, top_k=6,
             tokens=3001, max_tokens=4096, micro=1, skew=0.35),
        # decode with fp8 experts: the serving loop replays one graph per batch size
        dict(name="stack_fp8_64", kind="stack", mode="infer", fp8=True, graph=True, experts=32, tokens=64, max_tokens=4096,
             skew=0.7),
        # prefill with fp8 experts
        dict(name="stack_fp8_4096", kind="stack", mode="infer", fp8=True, graph=False, experts=32, tokens=4096,
             max_tokens=4096, skew=0.7),
        # the largest: a training step of the DeepSeek-V3-shaped block
        dict(name="stack_step_4096", kind="stack", mode="step", fp8=False, graph=False, experts=32, tokens=4096,
             max_tokens=4096, skew=0.7),
        # a step of the GPT: one layer of the recipe, dense parts included
        dict(name="gpt_step_4096", kind="gpt", layers=1, hidden=2048, heads=16, ffn=1024, experts=64, top_k=8, vocab=32000,
             seq=2048, batch=2, skew=0.35),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _layer_shape(rng, names):
    """A recipe's expert shape, or (one in four) a generic one within the kernels' documented multiples."""
    if rng.random() < 0.25:
        return dict(hidden=64 * rng.randint(8, 40), ffn=128 * rng.randint(3, 12), experts=rng.choice([8, 16, 24, 40, 64, 96]),
                    top_k=rng.randint(1, 8))
    name = rng.choice(names)
    if name == "bench":
        return dict(hidden=2048, ffn=1408, experts=64, top_k=6)
    r = RECIPES[name]
    return dict(hidden=r["hidden"], ffn=r["ffn"], experts=r["experts"], top_k=r["top_k"])


def draw(rng):
    kind = rng.choice(["plan", "layer", "layer", "layer_infer", "layer_infer", "stack", "stack", "gpt"])
    skew = round(rng.uniform(0.0, 0.8), 3)
    if kind == "plan":
        domains, per_domain = rng.choice([(1, 8), (2, 4), (4, 2), (2, 8), (4, 8), (8, 8)])
        per_rank = max(1, _log_int(rng, 32, 512) // (domains * per_domain))
        return dict(kind="plan", experts=per_rank * domains * per_domain, domains=domains, per_domain=per_domain,
                    extra=rng.choice([1, 2, 4]), skew=round(rng.uniform(1.0, 1.5), 3), top_k=rng.choice([4, 6, 8]))
    if kind == "layer":
        shape = _layer_shape(rng, ["bench", "gpt_moe_1b", "qwen3_30b_a3b", "tiny"])
        tokens = _log_int(rng, 33, 8192)
        accum = rng.random() < 0.3
        return dict(kind="layer", mode="step", graph=not accum and rng.random() < 0.5, tokens=tokens,
                    max_tokens=min(8192, tokens + rng.choice([0, 1, 300])), micro=2 if accum else 1, skew=skew, **shape)
    if kind == "layer_infer":
        shape = _layer_shape(rng, ["bench", "gpt_moe_1b", "qwen3_30b_a3b", "glm45_air", "deepseek_v2_160e"])
        tokens = _log_int(rng, 1, 8192)
        return dict(kind="layer", mode="infer", graph=rng.random() < 0.5, tokens=tokens, max_tokens=max(tokens, rng.choice([512, 4096])),
                    micro=1, skew=skew, **shape)
    if kind == "stack":
        mode = rng.choice(["infer", "infer", "infer", "step"])
        tokens = _log_int(rng, 1 if mode == "infer" else 64, 4095)
        return dict(kind="stack", mode=mode, fp8=mode == "infer" and rng.random() < 0.75, graph=mode == "infer" and rng.random() < 0.5,
                    experts=rng.choice([16, 32]), tokens=tokens, max_tokens=max(tokens, rng.choice([512, 4096])), skew=skew)
    return dict(kind="gpt", layers=1, hidden=2048, heads=16, ffn=rng.choice([768, 1024]),
                experts=rng.choice([32, 64]), top_k=8, vocab=32000, seq=64 * rng.randint(4, 32), batch=rng.randint(1, 3), skew=skew)


# ---------------------------------------------------------------------- states
def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEVICE).to(torch.bfloat16)


def _held(tensor, owner):
    """``tensor`` of ``owner``'s symmetric memory as an output: the memory lives as long as its owner does."""
    out = tensor.detach()
    out.owner = owner
    return out


def _expert_outputs(out, moe, index=""):
    for name in ("w1", "w2"):
        p = getattr(moe, name)
        grad = getattr(p, "main_grad", None)
        out[f"{name}{index}"] = _held(p, moe.heap)
        out[f"{name}{index}_grad"] = _held(p.grad if grad is None else grad, moe.heap)


def _program(step_fn, x, graph):
    """One pass of ``step_fn`` on ``x``: launched eagerly, or replayed from a graph.  The graph works on memory that
    ``step_fn``'s model and optimizer own, so the pass keeps them."""
    step = GraphedStep(step_fn, x) if graph else step_fn

    def once():
        return step(x)

    once.program = step_fn
    return once


def _prepare_plan(c, seed):
    ranks, experts = c["domains"] * c["per_domain"], c["experts"]
    topo = Topology.from_nvlink_rdma(c["domains"], c["per_domain"]).to(DEVICE)
    spec = ProblemSpec.contiguous_main_placement(experts, ranks, 3 * 2048 * 1408 * 2, 2 * 2048, experts // ranks + c["extra"]).to(DEVICE)
    loads = make_loads(ranks, experts, 4096, c["top_k"], c["skew"], 0.25, seed, device=DEVICE)
    cfg = EPLBConfig()

    def once():
        plan = solve(loads, topo, spec, cfg, validate=False)
        return {"x": plan.x, "q": plan.q, "theta": plan.theta}

    return once


def _prepare_layer(c, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    accum = c["micro"] > 1
    cfg = MoEConfig(hidden=c["hidden"], ffn=c["ffn"], num_experts=c["experts"], top_k=c["top_k"], max_tokens=c["max_tokens"],
                    grad_accum_dtype=torch.float32 if accum else None)
    layer = FusedMoE(cfg, SymmetricHeap(heap_layout(cfg, 1), torch.device(DEVICE)), 0, 1, seed=seed)
    layer.router_bias = c["skew"] * torch.randn(c["experts"], generator=gen, device=DEVICE)
    batches = [_randn(gen, c["tokens"], c["hidden"]) for _ in range(c["micro"])]

    if c["mode"] == "infer":
        @torch.no_grad()
        def forward(x):
            return {"out": layer(x)}

        return _program(forward, batches[0], c["graph"])

    opt = FusedAdamW(layer.parameters(), lr=1e-5, capturable=c["graph"], guard=layer.loc["status"].view(1, 4))

    def outputs(out, x, **more):
        res = dict(out=out.detach(), dx=x.grad, router=layer.router.detach(), router_grad=layer.router.grad, **more)
        _expert_outputs(res, layer)
        return res

    if not accum:  # the README's step
        def train(x):
            x = x.detach().requires_grad_(True)
            opt.zero_grad(set_to_none=True)
            out = layer(x)
            loss = out.float().square().mean()
            loss.backward()
            opt.step()
            return outputs(out, x, loss=loss.detach())

        return _program(train, batches[0], c["graph"])

    douts = [_randn(gen, c["tokens"], c["hidden"]) for _ in batches]

    def micro_batches():
        opt.zero_grad(set_to_none=True)
        layer.zero_grad_accum()
        for b, dout in zip(batches, douts):
            x = b.detach().requires_grad_(True)
            out = layer(x)
            out.backward(dout)
        opt.step()
        return outputs(out, x)

    return micro_batches


def _prepare_stack(c, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    torch.manual_seed(seed)
    cfg = DSv3Config(layers=1, experts=c["experts"], max_tokens=c["max_tokens"], num_domains=1, fp8_inference=c["fp8"], **STACK)
    model = DSv3Stack(cfg, torch.device(DEVICE))
    model.set_router_bias(c["skew"] * torch.randn(1, c["experts"], generator=gen, device=DEVICE))
    x0 = _randn(gen, c["tokens"], cfg.hidden)
    if c["mode"] == "infer":
        if c["fp8"]:
            model.quantize_weights()

        @torch.no_grad()
        def forward(x):
            return {"out": model(x)}

        return _program(forward, x0, c["graph"])

    dense_opt = FusedAdamW(model.dense_parameters(), lr=1e-5, guard=model.status.words)
    expert_opt = FusedAdamW(list(model.expert_parameters()), lr=1e-5, guard=model.status.words)
    dout = _randn(gen, c["tokens"], cfg.hidden)
    moe, shared = model.blocks[0].moe, model.blocks[0].shared

    def train():
        dense_opt.zero_grad(set_to_none=True)
        x = x0.detach().requires_grad_(True)
        out = model(x)
        out.backward(dout)
        dense_opt.step()
        expert_opt.step()
        res = dict(out=out.detach(), dx=x.grad, router=moe.router.detach(), router_grad=moe.router.grad,
                   shared_up=shared.up.weight.detach(), shared_up_grad=shared.up.weight.grad,
                   shared_down=shared.down.weight.detach(), shared_down_grad=shared.down.weight.grad)
        _expert_outputs(res, moe)
        return res

    return train


def _prepare_gpt(c, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    torch.manual_seed(seed)
    cfg = GPTMoEConfig(vocab=c["vocab"], layers=c["layers"], hidden=c["hidden"], heads=c["heads"], ffn=c["ffn"], experts=c["experts"],
                       top_k=c["top_k"], seq_len=c["seq"], micro_batch=c["batch"])
    model = GPTMoE(cfg, torch.device(DEVICE))
    model.set_router_bias(c["skew"] * torch.randn(c["layers"], c["experts"], generator=gen, device=DEVICE))
    dense_opt = FusedAdamW(model.dense_parameters(), lr=1e-5, guard=model.status.words)
    expert_opt = FusedAdamW(list(model.expert_parameters()), lr=1e-5, guard=model.status.words)
    ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=gen, device=DEVICE)

    def train():
        dense_opt.zero_grad(set_to_none=True)
        loss = model(ids[:, :-1], ids[:, 1:])
        loss.backward()
        dense_opt.step()
        expert_opt.step()
        res = {"loss": loss.detach(), "embed_grad": model.embed.weight.grad, "head_grad": model.head.weight.grad}
        for i, b in enumerate(model.blocks):
            res[f"qkv{i}_grad"], res[f"router{i}_grad"] = b.attn.qkv.weight.grad, b.moe.router.grad
            _expert_outputs(res, b.moe, i)
        return res

    return train


_PREPARE = {"plan": _prepare_plan, "layer": _prepare_layer, "stack": _prepare_stack, "gpt": _prepare_gpt}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return state()


# ---------------------------------------------------------------------- what a pass cannot do without
def _adam_bytes(params, grad_bytes=2):
    """Parameter and both moments (bf16) read and written, the gradient read."""
    return params * (12 + grad_bytes)


def _moe_work(tokens, hidden, ffn, experts, top_k, weight_bytes, train):
    """Forward (and backward): router and three expert projections; inputs, weights and outputs once."""
    units = tokens * top_k
    used = min(experts, units)
    flops = 2 * tokens * hidden * experts + 6 * units * hidden * ffn
    nbytes = 2 * 2 * tokens * hidden + used * 3 * hidden * ffn * weight_bytes + 4 * experts * hidden
    if train:
        flops *= 3
        nbytes += 2 * 2 * tokens * hidden + used * 3 * hidden * ffn * 2 + experts * 3 * hidden * ffn * 2 + 8 * experts * hidden
    return flops, nbytes


def work(case):
    c = case
    if c["kind"] == "plan":
        ranks, experts = c["domains"] * c["per_domain"], c["experts"]
        return {"bytes": 8 * ranks * experts + experts * ranks + 8 * ranks * experts * ranks, "flops": 0}
    train = c.get("mode", "step") == "step"
    if c["kind"] == "layer":
        flops, nbytes = _moe_work(c["tokens"], c["hidden"], c["ffn"], c["experts"], c["top_k"], 2, train)
        if train:
            params = c["experts"] * 3 * c["hidden"] * c["ffn"]
            flops, nbytes = flops * c["micro"], nbytes * c["micro"] + _adam_bytes(params, 4 if c["micro"] > 1 else 2)
        return {"bytes": nbytes, "flops": flops}
    if c["kind"] == "stack":
        H, F = STACK["hidden"], STACK["ffn"]
        flops, nbytes = _moe_work(c["tokens"], H, F, c["experts"], 8, 1 if c["fp8"] else 2, train)
        dense = 3 * H * F
        flops += 2 * c["tokens"] * dense * (3 if train else 1)
        nbytes += 2 * dense * (3 if train else 1)
        if train:
            nbytes += _adam_bytes(dense + c["experts"] * 3 * H * F)
        return {"bytes": nbytes, "flops": flops}
    tokens, H = c["seq"] * c["batch"], c["hidden"]
    flops, nbytes = _moe_work(tokens, H, c["ffn"], c["experts"], c["top_k"], 2, True)
    dense = 4 * H * H
    flops += 3 * (2 * tokens * dense + 2 * tokens * c["seq"] * H)
    flops, nbytes = flops * c["layers"], (nbytes + 6 * dense) * c["layers"]
    flops += 3 * 2 * tokens * H * c["vocab"]
    params = c["layers"] * (dense + c["experts"] * 3 * H * c["ffn"]) + 2 * c["vocab"] * H
    return {"bytes": nbytes + 6 * 2 * c["vocab"] * H + _adam_bytes(params), "flops": flops}


def tolerance(case):
    """The plan is whole numbers that every rank has to agree on.  The rest was compared, output by output, with the same
    pass in plain PyTorch with fp32 sums: bf16 layers are off by up to 5.8e-3 (weight gradients), fp8 blocks by 9.3e-3 (a
    pre-activation that rounds the other way moves a value to the next of three mantissa bits)."""
    if case["kind"] == "plan":
        return "exact"
    return {"rel": 3e-2 if case.get("fp8") else 2e-2}
