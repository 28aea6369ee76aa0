"""The launch sequences that FFM_OVERLAP=0 and FFM_FUSED_GLU_BACKWARD=0 select in the native driver, against the default."""

import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import MoELayer, ops  # noqa: E402

layer_module = importlib.import_module("flashfusedmoe_b200.fused_moe")
DEV = "cuda"
SCHEDULES = [(overlap, fused) for overlap in (True, False) for fused in (True, False)]


# a ragged step with few tokens; one whose shared down-projection's gradient is summed in two ranges of the tokens
@pytest.mark.parametrize("N", [300, 8200])
@pytest.mark.parametrize("options", [dict(num_shared_experts=1, aux_loss_coeff=0.01, z_loss_coeff=0.001), dict(),
                                     dict(num_shared_experts=1, recompute_activations=True, gating="sigmoid",
                                          aux_loss_coeff=0.01), dict(capacity_factor=1.0, activation="geglu")])
def test_schedules_agree(N, options, monkeypatch):
    """Neither the side streams nor the place where the GLU backward runs changes a bit."""
    D = 256
    torch.manual_seed(N)
    layer = MoELayer(D, 512, 8, 2, **options).to(DEV).bfloat16().train(True)
    x = torch.randn(N, D, device=DEV).bfloat16().requires_grad_(True)
    go = torch.randn(N, D, device=DEV).bfloat16()
    names, leaves = zip(*[("x", x), *layer.named_parameters()])
    results = {}
    for schedule in SCHEDULES:
        monkeypatch.setattr(layer_module, "_OVERLAP", schedule[0])
        monkeypatch.setattr(layer_module, "_FUSED_GLU_BWD", schedule[1])
        out, losses = layer(x)
        scalars = [losses[n] for n in ("aux_loss", "z_loss") if n in losses]
        grads = torch.autograd.grad([out, *scalars], leaves, [go, *[torch.ones_like(s) for s in scalars]])
        ops.check_status()
        results[schedule] = dict(zip(names, grads), out=out.detach(), **{f"loss{i}": s.detach() for i, s in enumerate(scalars)})
    want = results[True, True]
    for schedule, got in results.items():
        for name in got:
            assert torch.equal(got[name], want[name]), (schedule, name)
