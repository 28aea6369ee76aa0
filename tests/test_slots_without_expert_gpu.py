"""A token whose scores are NaN has no expert: its slots get defined marks, its rows are NaN, every other token is as without
it, and the failure is reported."""

import pytest
import torch

pytestmark = pytest.mark.gpu

import flashfusedmoe_b200 as ffm  # noqa: E402
from flashfusedmoe_b200 import ops  # noqa: E402

DEV = "cuda"


def _inputs(N, D, E, bad):
    g = torch.Generator(device=DEV).manual_seed(N + E)
    hidden = torch.randn(N, D, generator=g, device=DEV).bfloat16()
    gate = torch.randn(E, D, generator=g, device=DEV).bfloat16()
    broken = hidden.clone()
    broken[bad] = float("nan")
    return hidden, broken, gate


# few tokens (one block, a cluster), then more: 8, 16 and 32 lanes per token, the tensor-core gate, the shared gate
@pytest.mark.parametrize("N,D,E,k", [(5, 64, 8, 2), (100, 128, 64, 6), (300, 128, 8, 2), (300, 72, 16, 4), (300, 64, 24, 3),
                                     (300, 64, 64, 6), (300, 72, 72, 4)])
@pytest.mark.parametrize("gating", ["softmax", "sigmoid"])
def test_routing_marks_them(N, D, E, k, gating):
    bad = [0, N - 2]
    hidden, broken, gate = _inputs(N, D, E, bad)
    want = ops.route_forward(hidden, gate, k, gating)
    ops.check_status()
    got = ops.route_forward(broken, gate, k, gating)
    with pytest.raises(RuntimeError, match="status"):
        ops.check_status()
    ok = torch.ones(N, dtype=torch.bool, device=DEV)
    ok[bad] = False
    assert torch.equal(got.topk_idx[ok], want.topk_idx[ok]) and torch.equal(got.topk_w[ok], want.topk_w[ok])
    assert bool((got.topk_idx[~ok] == -1).all()) and bool((got.pos.view(N, k)[~ok] == -1).all())
    flat = got.topk_idx.long()[ok].view(-1)
    assert torch.equal(got.counts.long(), torch.bincount(flat, minlength=E))
    slots = torch.arange(N * k, device=DEV).view(N, k)[ok].view(-1)
    assert torch.equal(got.src.long()[got.pos.view(N, k)[ok].long().view(-1)], slots)
    assert int((got.src >= 0).sum()) == slots.numel()
    cpos, src_c = ops.compact_positions(got, N * k)
    assert torch.equal(cpos >= 0, got.pos >= 0)
    rows = slots.numel()
    assert torch.equal(src_c.long()[cpos.long()[slots]], slots) and bool((src_c[rows:] == -1).all())


@pytest.mark.parametrize("weighted", [False, True])
def test_combine_without_a_row(weighted):
    N, D, k = 37, 264, 3
    Y = torch.randn(N * k, D, device=DEV).bfloat16()
    pos = torch.randperm(N * k, device=DEV).to(torch.int32)
    w = torch.rand(N, k, device=DEV) if weighted else None
    want = ops.combine_forward(Y, pos, w, N, k)
    holes = pos.clone()
    holes[3 * k + 1] = -1
    holes[20 * k:21 * k] = -1
    got = ops.combine_forward(Y, holes, w, N, k, addend=torch.zeros_like(want))
    bad = torch.zeros(N, dtype=torch.bool, device=DEV)
    bad[[3, 20]] = True
    assert torch.equal(got[~bad], want[~bad]) and bool(got[bad].isnan().all())


@pytest.mark.parametrize("gating", ["softmax", "sigmoid"])
@pytest.mark.parametrize("N", [40, 300])
def test_layer_reports_and_contains_them(N, gating):
    """Forward and input gradient of the other tokens: the bits they have without the bad token's contents."""
    D, E, k = 128, 8, 2
    bad = [7]
    hidden, broken, gate = _inputs(N, D, E, bad)
    g = torch.Generator(device=DEV).manual_seed(1)
    w_up, w_down = ((torch.randn(*s, generator=g, device=DEV) * 0.05).bfloat16() for s in ((E, 256, D), (E, D, 128)))
    go = torch.randn(N, D, generator=g, device=DEV).bfloat16()
    res = []
    for h in (hidden, broken):
        h = h.clone().requires_grad_(True)
        out, losses = ffm.fused_moe(h, gate, w_up, w_down, top_k=k, gating=gating)
        out.backward(go)
        res.append((out.detach(), h.grad))
    with pytest.raises(RuntimeError, match="status"):
        ops.check_status()
    ok = torch.ones(N, dtype=torch.bool, device=DEV)
    ok[bad] = False
    for want, got in zip(*res):
        assert torch.equal(got[ok], want[ok]) and bool(got[~ok].isnan().all())
    ffm.fused_moe(hidden, gate, w_up, w_down, top_k=k)
    ops.check_status()
