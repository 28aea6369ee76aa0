"""The layer's kernels follow one another: with a shared expert a call gives the bits of the same kernels launched one by one (without
one: test_chained_launches_gpu.py), and no kernel of a captured call may start before the ones it depends on have ended."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import MoELayer, _lib, ops  # noqa: E402

DEV = "cuda"


def _one_by_one(x, g, wu, wd, k, shared):
    N, D = x.shape
    E, H = wu.shape[0], wu.shape[1] // 2
    r = ops.route_forward(x, g, k)
    Xg = ops.permute_rows(x, r.src, ops.rows_capacity(N * k, E), k)
    act, _ = ops.grouped_gemm_glu(Xg, wu, wu.view(-1, D)[H:], 2 * H, E, r.tile_start, D, H, "swiglu", want_preact=False)
    Y = ops.grouped_gemm(act, wd, _lib.B_KMAJOR, E, r.tile_start, H, D)
    gate, up, down = shared
    s_act, _ = ops.grouped_gemm_glu(x, gate, up, gate.shape[0], 1, None, D, gate.shape[0], "swiglu", want_preact=False)
    add = ops.grouped_gemm(s_act, down, _lib.B_KMAJOR, 1, None, gate.shape[0], D)
    return ops.combine_forward(Y, r.pos, r.topk_w, N, k, add)


# the shared expert inside the one chain, and beside the routing on its own stream
@pytest.mark.parametrize("N", [5, 300, 4001])
def test_shared_expert_against_single_launches(N):
    torch.manual_seed(N)
    layer = MoELayer(256, 1024, 8, 2, num_shared_experts=1).to(DEV).bfloat16().eval()
    shared = [getattr(layer.shared_expert, name).weight for name in ("w_gate", "w_up", "w_down")]
    xs = [torch.randn(N, 256, device=DEV).bfloat16() for _ in range(12)]
    with torch.no_grad():
        want = [_one_by_one(x, layer.gate.weight, layer.w_up, layer.w_down, 2, shared) for x in xs]
        torch.cuda.synchronize()
        got = [layer(x)[0] for x in xs]
    ops.check_status()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


class _Edge(ctypes.Structure):   # CUgraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte),
                ("reserved", ctypes.c_ubyte * 5)]


# one chain; a prompt beside a shared expert; a training step, and one that recomputes
@pytest.mark.parametrize("N,train,recompute", [(1, False, False), (300, False, False), (300, True, False), (300, True, True)])
def test_captured_call_has_only_full_dependencies(N, train, recompute):
    """Every edge of the captured call waits for the end of the kernel before: no other kind is ordered with what a program, or
    the allocator, puts between two of the call's launches."""
    torch.manual_seed(0)
    layer = MoELayer(256, 512, 8, 2, num_shared_experts=1, recompute_activations=recompute).to(DEV).bfloat16().train(train)
    x = torch.randn(N, 256, device=DEV).bfloat16().requires_grad_(train)
    go = torch.randn(N, 256, device=DEV).bfloat16()

    def step():
        with torch.set_grad_enabled(train):
            out = layer(x)[0]
        return torch.autograd.grad(out, [x, *layer.parameters()], go) if train else out

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        kept = step()
    driver = ctypes.CDLL("libcuda.so.1")
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert driver.cuGraphGetEdges_v2(handle, None, None, None, ctypes.byref(n)) == 0
    assert n.value >= 4
    nodes, edges = ctypes.c_void_p * n.value, (_Edge * n.value)()
    assert driver.cuGraphGetEdges_v2(handle, nodes(), nodes(), edges, ctypes.byref(n)) == 0
    assert all((e.from_port, e.to_port, e.type) == (0, 0, 0) for e in edges)
    del kept
