"""ops.launch_count is the number of this library's kernels in a call: compared with the kernel nodes of the captured call."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import MoELayer, ops  # noqa: E402

DEV = "cuda"
KERNEL_NODE = 0   # CU_GRAPH_NODE_TYPE_KERNEL


def _kernel_nodes(graph):
    driver = ctypes.CDLL("libcuda.so.1")
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert driver.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes, kind = (ctypes.c_void_p * n.value)(), ctypes.c_int(-1)
    assert driver.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    kernels = 0
    for node in nodes:
        assert driver.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kernels += kind.value == KERNEL_NODE
    return kernels


# the one chain (5); more than a few tokens: the gate kernel, the tensor-core gate; a training step without and with a GEMM
# for the routing's input gradient, and with the shared down-projection's gradient in two ranges
@pytest.mark.parametrize("N,E,shared,train,z", [(1, 8, 1, False, 0.0), (300, 8, 1, False, 0.0), (300, 64, 0, False, 0.0),
                                                (300, 64, 1, True, 0.0), (300, 64, 0, True, 0.001), (8192, 64, 1, True, 0.001)])
def test_every_kernel_is_counted(N, E, shared, train, z):
    torch.manual_seed(0)
    layer = MoELayer(256, 512, E, 2, num_shared_experts=shared, z_loss_coeff=z).to(DEV).bfloat16().train(train)
    x = torch.randn(N, 256, device=DEV).bfloat16().requires_grad_(train)
    go = torch.randn(N, 256, device=DEV).bfloat16()
    one = torch.ones((), device=DEV)
    leaves = [x, *layer.parameters()]

    def step():
        if not train:
            with torch.no_grad():
                return layer(x)
        out, losses = layer(x)
        return torch.autograd.grad([out, *losses.values()], leaves, [go, *[one for _ in losses]])

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = ops.launch_count
    with torch.cuda.graph(graph):
        kept = step()
    counted = ops.launch_count - before
    assert counted == _kernel_nodes(graph)
    if N == 1:
        assert counted == 5
    del kept
