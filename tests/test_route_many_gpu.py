"""Routing of more than 256 tokens: every gate kernel and selection option, bit for bit against the path for few tokens and
its maps and statistics against torch."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import ops  # noqa: E402

DEV = "cuda"
FEW = 256

# D decides how many warps split a row (1, 2, 4, 8 with up to 32 experts), E the lanes per token (8, 16, 32) or the gate kernel:
# 33, 72, 129 experts, or D no multiple of 64, share a block's warps; 64 experts take the tensor-core gate. N gives ragged
# last blocks, and several trips per block where it exceeds 592 blocks of one trip (32, 16, 8 and 4 tokens for the four
# splits; 8, 4 and 2 for the shared gate).
SHAPES = [(257, 256, 8, 2, 4, 2), (20001, 256, 8, 4, 4, 3), (10003, 512, 16, 4, 8, 3), (5003, 264, 24, 6, 8, 3),
          (5003, 1024, 24, 3, 4, 1), (3001, 2056, 8, 2, 2, 1), (2501, 2048, 17, 4, 17, 4), (300, 72, 32, 6, 8, 2),
          (4999, 64, 33, 6, 11, 3), (2601, 72, 64, 8, 8, 4), (2501, 128, 72, 6, 8, 3), (1301, 64, 129, 8, 3, 2),
          (700, 72, 256, 8, 16, 4), (3001, 128, 64, 6, 8, 3)]


@pytest.mark.parametrize("opts", [dict(), dict(gating="sigmoid"), dict(pre_softmax=True, weight_scale=2.5),
                                  dict(groups=True), dict(gating="sigmoid", groups=True, weight_scale=0.5),
                                  dict(pre_softmax=True, groups=True)])
@pytest.mark.parametrize("N,D,E,k,n_group,topk_group", SHAPES)
def test_many_tokens_route_as_few(N, D, E, k, n_group, topk_group, opts):
    """Small integers: every logit is exact in any order of sums, so both paths must agree bit for bit."""
    opts = dict(opts)
    if opts.pop("groups", False):
        opts.update(n_group=n_group, topk_group=topk_group)
    g = torch.Generator(device=DEV).manual_seed(N + E)
    hidden = torch.randint(-2, 3, (N, D), generator=g, device=DEV).bfloat16()
    gate = (torch.randint(-2, 3, (E, D), generator=g, device=DEV) / 8).bfloat16()
    bias = torch.randn(E, generator=g, device=DEV)
    many = ops.route_forward(hidden, gate, k, expert_bias=bias, **opts)
    ops.check_status()
    assert torch.equal(many.logits, (hidden.float() @ gate.float().T).bfloat16())
    for n0 in sorted({0, (N // 2) // 8 * 8 + 3, N - FEW}):
        few = ops.route_forward(hidden[n0:n0 + FEW].contiguous(), gate, k, expert_bias=bias, **opts)
        for name in ("topk_idx", "topk_w", "lse"):
            assert torch.equal(getattr(few, name), getattr(many, name)[n0:n0 + FEW]), (name, n0)
    ops.check_status()

    flat = many.topk_idx.long().view(-1)
    counts = torch.bincount(flat, minlength=E)
    assert torch.equal(many.counts.long(), counts)
    tiles = torch.div(counts + 255, 256, rounding_mode="floor") * 2
    start = torch.cat([tiles.new_zeros(1), tiles.cumsum(0)])
    assert torch.equal(many.tile_start.long(), start)
    order = torch.sort(flat, stable=True).indices
    rank = torch.empty_like(order)
    rank[order] = torch.arange(N * k, device=DEV) - (counts.cumsum(0) - counts)[flat[order]]
    pos = start[flat] * 128 + rank
    assert torch.equal(many.pos.long(), pos)
    src = torch.full((many.rows_cap,), -1, dtype=torch.long, device=DEV)
    src[pos] = torch.arange(N * k, device=DEV)
    assert torch.equal(many.src.long()[:many.rows_cap], src)

    # fp32 sums of N positive terms in another order: at most N ulp apart, in practice a few; scores from fast exponentials
    # are within 1e-6 of torch's
    if opts.get("gating") == "sigmoid":
        mass = torch.sigmoid(many.logits.double()).sum(0)
    else:
        mass = torch.zeros(E, dtype=torch.double, device=DEV).scatter_add_(0, flat, many.topk_w.double().view(-1))
    torch.testing.assert_close(many.stats[:E].double(), mass, rtol=1e-5, atol=1e-5)
    z = torch.logsumexp(many.logits.double(), 1).square().sum()
    torch.testing.assert_close(many.stats[E].double(), z, rtol=2e-5, atol=0)
    dot = (counts.double() * many.stats[:E].double()).sum()
    torch.testing.assert_close(many.stats[E + 1].double(), dot, rtol=1e-5, atol=0)
