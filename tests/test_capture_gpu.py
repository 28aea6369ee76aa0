"""The layer under CUDA graph capture: the side streams that a call forks are joined before it returns, so a step can be
captured, and its replay gives the same bits as the eager step, also for new values in the same buffers."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import MoELayer, ops  # noqa: E402

DEV = "cuda"


# training with a shared expert and both losses (all five streams; a split shared weight gradient from 8192 tokens on),
# recomputed, inference beside the shared expert, and the one-chain decode
@pytest.mark.parametrize("N,grad,recompute", [(300, True, False), (8192, True, False), (300, True, True), (300, False, False),
                                              (5, False, False)])
def test_replay_equals_eager(N, grad, recompute):
    torch.manual_seed(N)
    layer = MoELayer(256, 512, 8, 2, num_shared_experts=1, aux_loss_coeff=0.01, z_loss_coeff=0.001,
                     recompute_activations=recompute).to(DEV).bfloat16().train(grad)
    x = torch.randn(N, 256, device=DEV).bfloat16().requires_grad_(grad)
    go = torch.randn(N, 256, device=DEV).bfloat16()
    one = torch.ones((), device=DEV)
    leaves = [x, *layer.parameters()]

    def step():
        if not grad:
            with torch.no_grad():
                return [layer(x)[0]]
        out, losses = layer(x)
        return [out.detach(), *torch.autograd.grad([out, losses["aux_loss"], losses["z_loss"]], leaves, [go, one, one])]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(2):
        with torch.no_grad():
            x.copy_(torch.randn(N, 256, device=DEV).bfloat16())
        graph.replay()
        torch.cuda.synchronize()
        want = step()
        ops.check_status()
        for a, b in zip(captured, want):
            assert torch.equal(a, b)
