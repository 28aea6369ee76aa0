"""The layer calls whose speed is watched, over the sizes the layer is used at.

A case is one call a user's program makes: a training step (forward and backward, gradients of the tokens and of every
weight), a prefill (forward without gradients over many tokens) or a decode step (the same over few tokens). The shapes
are the ones the repository benchmarks and tests, and shapes between them: one row per family below.
"""

import math

import torch

from flashfusedmoe_b200 import MoELayer, fused_moe, set_expert_gemm_precision

# family: d_model, ffn_dim (gate and up together), experts, top_k, shared expert's ffn_dim (0: none)
FAMILIES = {
    "small": (256, 1024, 8, 2, 0),       # plumbing-sized layer of the tests
    "layer": (1024, 4096, 8, 2, 4096),   # the benchmark's layer: 8 experts and a shared one
    "wide": (4096, 28672, 8, 2, 0),      # few wide experts, called through fused_moe() with a skewed expert bias
    "fine": (2048, 2816, 64, 6, 5632),   # fine-grained experts, two shared ones merged into one
    "many": (7168, 4096, 256, 8, 4096),  # 256 experts: 22.5 GB of weights, inference only
    "mid": (1024, 2816, 16, 4, 0),       # between "layer" and "fine"
}


def _case(kind, family, tokens, **options):
    d, f, e, k, s = FAMILIES[family]
    case = dict(kind=kind, d_model=d, ffn_dim=f, experts=e, top_k=k, shared_ffn=s, tokens=tokens, activation="swiglu",
                gating="softmax", aux=0.0, z=0.0, recompute=False, autocast=False, fp8=False, skew=False)
    case.update(options)
    return case


def listed():
    def named(name, *a, **o):
        return dict(_case(*a, **o), name=name)

    return [
        # one sequence of chat, one token at a time: nothing but latency and launches
        named("decode_layer_1", "decode", "layer", 1),
        # a small batch of sequences on fine-grained experts
        named("decode_fine_48", "decode", "fine", 48),
        # a handful of sequences on few wide experts: the weights that are hit are streamed once
        named("decode_wide_7", "decode", "wide", 7, skew=True),
        # a serving batch on 256 experts: nearly every expert is hit by a few rows
        named("decode_many_128", "decode", "many", 128),
        # one prompt of odd length
        named("prefill_layer_1999", "prefill", "layer", 1999),
        # a batch of prompts on fine-grained experts
        named("prefill_fine_4096", "prefill", "fine", 4096),
        # a batch of prompts with the e4m3 forward projections
        named("prefill_layer_fp8_8192", "prefill", "layer", 8192, fp8=True),
        # a debugging-sized training step, fp32 parameters under autocast, both losses
        named("train_small_512_autocast", "train", "small", 512, autocast=True, aux=0.01, z=0.001),
        # a ragged micro-batch with sigmoid gating, GEGLU and recomputed activations
        named("train_mid_3001", "train", "mid", 3001, gating="sigmoid", activation="geglu", aux=0.01, recompute=True),
        # the benchmark's training step, with the load-balance loss that training switches on
        named("train_layer_16384", "train", "layer", 16384, aux=0.01),
        # a training step on fine-grained experts
        named("train_fine_16384", "train", "fine", 16384, aux=0.01, z=0.001),
        # a training step on few wide experts with an imbalanced load: the largest amount of arithmetic
        named("train_wide_8192", "train", "wide", 8192, skew=True),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["decode", "prefill", "train"])
    family = rng.choice(["small", "layer", "fine", "mid", "wide"])
    d, f, e, k, s = FAMILIES[family]
    if rng.random() < 0.5:  # a shape beside the family's
        d = 64 * max(2, round(d / 64 * rng.uniform(0.6, 1.1)))
        f = 128 * max(2, round(f / 128 * rng.uniform(0.6, 1.1)))
        s = 128 * round(s / 128 * rng.uniform(0.6, 1.1))
    tokens = {"decode": log_int(1, 192), "prefill": log_int(256, 16384), "train": log_int(64, 16384)}[kind]
    if family == "wide":
        tokens = min(tokens, 6000 + rng.randrange(1000))
    case = _case(kind, family, tokens, skew=rng.random() < 0.3)
    case.update(d_model=d, ffn_dim=f, shared_ffn=s)
    case["gating"] = rng.choice(["softmax", "softmax", "sigmoid"])
    case["activation"] = rng.choice(["swiglu", "swiglu", "geglu", "relu_squared"])
    if kind == "train":
        case["aux"] = rng.choice([0.0, 0.01])
        case["z"] = rng.choice([0.0, 0.001])
        case["recompute"] = rng.random() < 0.25
        case["autocast"] = family != "wide" and rng.random() < 0.25
    elif kind == "prefill" and d % 128 == 0 and f % 256 == 0:
        case["fp8"] = rng.random() < 0.25
    return case


def _skewed_bias(experts, generator, device):
    """log of Zipf(1.1) shares over the experts in random order: selects with an imbalanced load."""
    share = 1.0 / torch.arange(1, experts + 1, dtype=torch.float32, device=device) ** 1.1
    bias = torch.log(share / share.sum())[torch.randperm(experts, generator=generator, device=device)]
    return bias - bias.mean()


def prepare(case, seed):
    device = torch.device("cuda")
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    d, f, e, k, n = (case[key] for key in ("d_model", "ffn_dim", "experts", "top_k", "tokens"))
    train = case["kind"] == "train"
    dtype = torch.float32 if case["autocast"] else torch.bfloat16

    def normal(*shape, std=1.0):
        return torch.empty(*shape, dtype=dtype, device=device).normal_(0.0, std, generator=g)

    state = dict(case)
    if case["skew"]:
        state["bias"] = _skewed_bias(e, g, device)
        state["weights"] = [w.requires_grad_(train) for w in
                            (normal(e, d, std=0.02), normal(e, f, d, std=0.02), normal(e, d, f // 2, std=0.02))]
    else:
        with torch.device("meta"):
            layer = MoELayer(d, f, e, k, activation=case["activation"], gating=case["gating"],
                             num_shared_experts=1 if case["shared_ffn"] else 0, shared_ffn_dim=case["shared_ffn"] or None,
                             aux_loss_coeff=case["aux"], z_loss_coeff=case["z"], recompute_activations=case["recompute"])
        layer = layer.to(dtype).to_empty(device=device)
        with torch.no_grad():
            for p in layer.parameters():
                p.normal_(0.0, 0.02, generator=g)
        state["layer"] = layer.train(train)
        state["weights"] = list(layer.parameters())
    state["x"] = normal(n, d).requires_grad_(train)
    if train:
        state["grad_out"] = torch.empty(n, d, dtype=torch.bfloat16, device=device).normal_(generator=g)
    return state


def _forward(state):
    if "layer" in state:
        return state["layer"](state["x"])
    gate, up, down = state["weights"]
    return fused_moe(state["x"], gate, up, down, top_k=state["top_k"], activation=state["activation"],
                     gating=state["gating"], aux_loss_coeff=state["aux"], z_loss_coeff=state["z"],
                     recompute_activations=state["recompute"], expert_bias=state["bias"])


def run(state):
    if state["kind"] == "train":
        leaves = [state["x"], *state["weights"]]
        for t in leaves:
            t.grad = None
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=state["autocast"]):
            out, losses = _forward(state)
        extra = [losses[name] for name in ("aux_loss", "z_loss") if name in losses]
        torch.autograd.backward([out, *extra], [state["grad_out"], *[None for _ in extra]])
        return [out.detach(), *[t.detach() for t in extra], *[t.grad for t in leaves]]
    with torch.no_grad():
        if not state["fp8"]:
            return _forward(state)[0]
        previous = set_expert_gemm_precision("fp8")
        try:
            return _forward(state)[0]
        finally:
            set_expert_gemm_precision(previous)


def work(case):
    d, f, e, k, n, s = (case[key] for key in ("d_model", "ffn_dim", "experts", "top_k", "tokens", "shared_ffn"))
    s = 0 if case["skew"] else s
    size = 4 if case["autocast"] else 2
    hit = e * (1.0 - (1.0 - k / e) ** n)  # experts that receive a row
    per_expert = 1.5 * f * d
    dense = 1.5 * s * d + e * d
    flops = 2.0 * n * k * per_expert + 2.0 * n * dense
    if case["kind"] != "train":
        return {"bytes": (hit * per_expert + dense) * size + 4.0 * n * d, "flops": flops}
    # weights read and their gradients written (of every expert), tokens, outputs and their gradients
    return {"bytes": (hit + e) * per_expert * size + 2.0 * dense * size + n * d * (2.0 * size + 4.0),
            "flops": 3.0 * flops}


_GATED = {
    "swiglu": torch.nn.functional.silu,
    "geglu": lambda g: torch.nn.functional.gelu(g, approximate="tanh"),
    "geglu_erf": torch.nn.functional.gelu,
    "relu_squared": lambda g: torch.relu(g).square(),
}


def exact(case, seed):
    """What run() returns, evaluated in 64 bits on the operands the layer computes with: parameters and tokens as bf16
    values, router logits rounded to bf16 (the layer's contract: experts are chosen on them, ties to the lower index),
    everything after that unrounded."""
    state = prepare(case, seed)
    train = case["kind"] == "train"
    if "layer" in state:
        names = [n for n, _ in state["layer"].named_parameters()]
    else:
        names = ["gate.weight", "w_up", "w_down"]
    given = dict(zip(names, state["weights"]))
    k, e, act = case["top_k"], case["experts"], case["activation"]
    h = case["ffn_dim"] // 2

    def wide(t):
        return t.detach().to(torch.bfloat16).double()

    x = wide(state["x"])
    n = x.shape[0]
    logits = (x @ wide(given["gate.weight"]).T).to(torch.bfloat16).double()
    value = logits if case["gating"] == "softmax" else torch.sigmoid(logits)
    select = value.float() + state["bias"] if "bias" in state else value
    idx = torch.sort(select, dim=1, descending=True, stable=True).indices[:, :k]
    leaf = logits.requires_grad_(train)
    picked = (leaf if case["gating"] == "softmax" else torch.sigmoid(leaf)).gather(1, idx)
    weight = torch.softmax(picked, 1) if case["gating"] == "softmax" else picked / (picked.sum(1, keepdim=True) + 1e-6)
    losses = []
    if train and case["aux"] > 0:
        f = torch.bincount(idx.reshape(-1), minlength=e).double() / n
        if case["gating"] == "softmax":
            share = torch.zeros(e, dtype=torch.float64, device=x.device).scatter_add(0, idx.reshape(-1), weight.reshape(-1)) / n
        else:
            share = torch.sigmoid(leaf).mean(0)
        losses.append(case["aux"] * e * (f * share).sum())
    if train and case["z"] > 0:
        losses.append(case["z"] * torch.logsumexp(leaf, 1).square().mean())
    out, go = torch.zeros_like(x), wide(state["grad_out"]) if train else None
    dx, dweight, grads = torch.zeros_like(x), torch.zeros_like(weight), {}

    def glu(rows, w_gate, w_up, w_down, g_rows, scale, activation):
        """GLU feed-forward of `rows`; with g_rows, the gradient of its scaled output, also every gradient."""
        a, u = rows @ w_gate.T, rows @ w_up.T
        if g_rows is None:
            return (_GATED[activation](a) * u) @ w_down.T, None
        a.requires_grad_(True)
        gated = _GATED[activation](a)
        hidden = (gated * u).detach()
        y = hidden @ w_down.T
        dy = g_rows * scale
        dhid = dy @ w_down
        da = torch.autograd.grad(gated, a, dhid * u)[0]
        du = dhid * gated.detach()
        return y, (da @ w_gate + du @ w_up, da.T @ rows, du.T @ rows, dy.T @ hidden)

    if train:
        grads["w_up"] = torch.zeros(given["w_up"].shape, dtype=torch.float64, device=x.device)
        grads["w_down"] = torch.zeros(given["w_down"].shape, dtype=torch.float64, device=x.device)
    for i in range(e):
        token, slot = torch.nonzero(idx == i, as_tuple=True)
        if token.numel() == 0:
            continue
        w = wide(given["w_up"][i])
        scale = weight.detach()[token, slot].unsqueeze(1)
        y, g = glu(x[token], w[:h], w[h:], wide(given["w_down"][i]), go[token] if train else None, scale, act)
        out.index_add_(0, token, y * scale)
        if train:
            dweight[token, slot] = (go[token] * y).sum(1)
            dx.index_add_(0, token, g[0])
            grads["w_up"][i, :h], grads["w_up"][i, h:], grads["w_down"][i] = g[1], g[2], g[3]
    if "shared_expert.w_gate.weight" in given:
        own = ["shared_expert.%s.weight" % m for m in ("w_gate", "w_up", "w_down")]
        y, g = glu(x, *(wide(given[m]) for m in own), go, 1.0, "geglu_erf" if act == "geglu" else act)
        out += y
        if train:
            dx += g[0]
            grads.update(zip(own, g[1:]))
    if not train:
        return out
    dlogits = torch.autograd.grad([(weight * dweight).sum(), *losses], leaf)[0]
    grads["gate.weight"] = dlogits.T @ x
    dx += dlogits @ wide(given["gate.weight"])
    return [out, *[t.detach() for t in losses], dx, *[grads[m] for m in names]]


def tolerance(case):
    # Against an fp32 evaluation with the same expert choice every output and gradient of the bf16 path lies within
    # rel 4.9e-3 and max 5.1e-2 (bf16 roundings of the pre-activations, activations, expert outputs and gradients in
    # turn); another order of roundings may differ by about three times that. e4m3 operands double the distance where
    # an activation rounds to its neighbour.
    return {"rel": 2e-2, "max": 0.2} if case["fp8"] else {"rel": 1.5e-2, "max": 0.15}
