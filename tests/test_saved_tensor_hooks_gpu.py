"""Saved-tensor hooks around the single-GPU layer: copies are used like the originals, and tensors that the native backward pass
cannot read are refused before it launches anything."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import MoELayer  # noqa: E402

DEV = "cuda"


def _step(unpack):
    torch.manual_seed(6)
    layer = MoELayer(128, 256, 8, 2, num_shared_experts=1).to(DEV).bfloat16().train(True)
    x = torch.randn(300, 128, device=DEV).bfloat16().requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        out = layer(x)[0]
    return torch.autograd.grad(out.float().square().sum(), [x, *layer.parameters()])


def test_copies():
    for got, want in zip(_step(lambda t: t.clone()), _step(lambda t: t)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.uint8, torch.int32])
@pytest.mark.parametrize("change,error", [(lambda t: t.cpu(), RuntimeError), (lambda t: t.double(), TypeError),
                                          (lambda t: torch.stack((t, t), -1)[..., 0], ValueError)])
def test_unreadable_tensors_are_refused(dtype, change, error):
    """Each kind of saved tensor (operands, routing results, counts) on the host, of another type, and not contiguous."""
    with pytest.raises(error, match="saved tensor"):
        _step(lambda t: change(t) if t.dtype == dtype else t)
