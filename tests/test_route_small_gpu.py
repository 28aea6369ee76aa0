"""Routing of few tokens (two launches) against the torch oracle, and against the kernels that route many tokens."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import ops  # noqa: E402
from test_kernels_gpu import test_route_forward as check_against_torch  # noqa: E402

DEV = "cuda"


# one block / a cluster, the last token group partly filled, expert groups of 8 and 16 partly filled, the line at 256
@pytest.mark.parametrize("N,D,E,k", [(1, 8, 1, 1), (2, 72, 9, 3), (15, 264, 17, 4), (16, 2056, 33, 6), (17, 128, 64, 6),
                                     (255, 64, 129, 8), (256, 64, 256, 16), (257, 64, 8, 2), (256, 64, 24, 17)])
def test_few_tokens(N, D, E, k):
    for gating in ("softmax", "sigmoid"):
        check_against_torch(N, D, E, k, gating)


@pytest.mark.parametrize("opts", [dict(), dict(gating="sigmoid"), dict(pre_softmax=True), dict(n_group=8, topk_group=3),
                                  dict(gating="sigmoid", n_group=4, topk_group=2, weight_scale=2.5)])
@pytest.mark.parametrize("N,E,k", [(5, 32, 4), (100, 64, 6), (256, 160, 8)])
def test_few_tokens_route_as_many(N, E, k, opts):
    """Small integers: every logit is exact in any order of sums, so both paths must agree bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(N + E)
    D = 256
    hidden = torch.randint(-2, 3, (N + 300, D), generator=g, device=DEV).bfloat16()
    gate = (torch.randint(-2, 3, (E, D), generator=g, device=DEV) / 8).bfloat16()
    bias = torch.randn(E, generator=g, device=DEV)
    few = ops.route_forward(hidden[:N].contiguous(), gate, k, expert_bias=bias, **opts)
    many = ops.route_forward(hidden, gate, k, expert_bias=bias, **opts)
    ops.check_status()
    for name in ("logits", "topk_w", "topk_idx", "lse"):
        assert torch.equal(getattr(few, name), getattr(many, name)[:N]), name
    flat = few.topk_idx.long().view(-1)
    assert torch.equal(few.counts.long(), torch.bincount(flat, minlength=E))
    assert torch.equal(few.src.long()[few.pos.long()], torch.arange(N * k, device=DEV))
    assert int((few.src >= 0).sum()) == N * k
    assert torch.equal(torch.div(few.pos.long(), 128, rounding_mode="floor") >= few.tile_start.long()[flat],
                       torch.ones_like(flat, dtype=torch.bool))
