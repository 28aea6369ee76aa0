"""Conversions between fp32 and bf16 of several tensors in one launch, against torch's own, and where the layer uses them."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import MoELayer, _lib, fused_moe, set_expert_gemm_precision  # noqa: E402
from flashfusedmoe_b200.fused_moe import glu_ffn  # noqa: E402

DEV = "cuda"


def _cast(tensors, dtype):
    out = [torch.full_like(t, float("nan"), dtype=dtype) for t in tensors]
    array = ctypes.c_int64 * len(tensors)
    src, dst, elements = (array(*v) for v in ([t.data_ptr() for t in tensors], [t.data_ptr() for t in out],
                                              [t.numel() for t in tensors]))
    rc = _lib.load().ffm_cast_many(len(tensors), src, dst, elements, int(dtype == torch.bfloat16),
                                   torch.cuda.current_stream().cuda_stream)
    return rc, out


@pytest.mark.parametrize("sizes", [(1,), (7, 8, 9), (0, 5, 0, 4097), (1, 2, 3, 4, 255, 256, 257, 70001), (3000001, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_cast_many(sizes, dtype):
    """Bit for bit torch's casts, at ends inside an eight-element chunk and with tensors without elements in between."""
    g = torch.Generator(device=DEV).manual_seed(sum(sizes))
    source = torch.float32 if dtype == torch.bfloat16 else torch.bfloat16
    tensors = [(torch.randn(n, generator=g, device=DEV) * 2.0 ** torch.randint(-100, 100, (n,), generator=g, device=DEV))
               .to(source) for n in sizes]
    tensors[-1][:1] = float("inf")
    rc, out = _cast(tensors, dtype)
    assert rc == 0
    for t, o in zip(tensors, out):
        assert torch.equal(o, t.to(dtype))


def test_cast_many_refuses():
    x = torch.zeros(64, device=DEV)
    assert _cast([x[1:]], torch.bfloat16)[0] != 0            # not on a 16-byte boundary
    assert _lib.load().ffm_cast_many(9, None, None, None, 1, None) != 0


@pytest.mark.parametrize("shared", [0, 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_fp32_parameters_under_autocast(shared, offset):
    """fp32 tokens and parameters give the results of the bf16 layer on the cast values, and its gradients as fp32; tokens off
    a 16-byte boundary or not contiguous are cast another way, with the same results."""
    torch.manual_seed(3)
    layer = MoELayer(128, 256, 8, 2, num_shared_experts=shared, aux_loss_coeff=0.01).to(DEV).train(True)
    narrow = MoELayer(128, 256, 8, 2, num_shared_experts=shared, aux_loss_coeff=0.01).to(DEV).bfloat16().train(True)
    narrow.load_state_dict(layer.state_dict())
    flat = torch.randn(300 * 128 + offset, device=DEV)
    x = flat[offset:].view(300, 128)
    go = torch.randn(300, 128, device=DEV).bfloat16()

    def step(m, tokens):
        tokens = tokens.detach().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out, losses = m(tokens)
        leaves = [tokens, *m.parameters()]
        return out, torch.autograd.grad([out, losses["aux_loss"]], leaves, [go, torch.ones((), device=DEV)]), leaves

    out, grads, leaves = step(layer, x)
    ref, ref_grads, _ = step(narrow, x.bfloat16())
    assert torch.equal(out, ref)
    for got, want, leaf in zip(grads, ref_grads, leaves):
        assert got.dtype == leaf.dtype and got.is_contiguous() and torch.equal(got, want.float())
    if offset == 0:
        wide = torch.randn(300, 256, device=DEV)
        wide[:, :128] = x
        out2, grads2, _ = step(layer, wide[:, :128])
        assert torch.equal(out2, ref) and torch.equal(grads2[0], grads[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tokens_whose_negation_is_pending(dtype):
    """A view may carry a negation that its memory does not hold (the imaginary part of a conjugate): it is carried out."""
    torch.manual_seed(4)
    layer = MoELayer(128, 256, 8, 2).to(DEV).to(dtype).eval()
    x = torch.randn(300, 128, device=DEV).to(dtype)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        want, got = layer(-x)[0], layer(torch._neg_view(x))[0]
    assert torch.equal(got, want)


# router alone; one half of the shared expert's gate and up; everything but that half and the router
@pytest.mark.parametrize("wide", [("gate.weight",), ("shared_expert.w_gate.weight",),
                                  ("w_up", "w_down", "shared_expert.w_up.weight", "shared_expert.w_down.weight")])
def test_layer_of_mixed_types(wide):
    """Some parameters fp32, the others bf16, on a stream that is not the default one: the bf16 layer's bits, each gradient in the
    type of its parameter."""
    torch.manual_seed(5)
    layer = MoELayer(128, 256, 8, 2, num_shared_experts=1, aux_loss_coeff=0.01).to(DEV).bfloat16().train(True)
    mixed = MoELayer(128, 256, 8, 2, num_shared_experts=1, aux_loss_coeff=0.01).to(DEV).bfloat16().train(True)
    mixed.load_state_dict(layer.state_dict())
    parameters = dict(mixed.named_parameters())
    for name in wide:
        parameters[name].data = parameters[name].data.float()
    x = torch.randn(300, 128, device=DEV).bfloat16()
    go = torch.randn(300, 128, device=DEV).bfloat16()

    def step(m):
        tokens = x.detach().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out, losses = m(tokens)
        leaves = [tokens, *m.parameters()]
        return out, torch.autograd.grad([out, losses["aux_loss"]], leaves, [go, torch.ones((), device=DEV)]), leaves

    ref, ref_grads, _ = step(layer)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        out, grads, leaves = step(mixed)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(out, ref)
    for got, want, leaf in zip(grads, ref_grads, leaves):
        assert got.dtype == leaf.dtype and torch.equal(got.float(), want.float())


def _negated(t):
    return torch._neg_view(t.neg())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_other_operands_whose_negation_is_pending(dtype):
    """The selection bias, the weights of the e4m3 projections, the gradients of the losses and a plain GLU block's operands."""
    torch.manual_seed(7)
    x = torch.randn(600, 128, device=DEV).bfloat16()
    g, wu, wd = (torch.randn(*s, device=DEV).mul_(0.05).to(dtype) for s in ((8, 128), (8, 512, 128), (8, 128, 256)))
    bias = torch.randn(8, device=DEV).to(dtype)

    def moe(*weights, expert_bias=None):
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return fused_moe(x, *weights, top_k=2, expert_bias=expert_bias)[0]

    assert torch.equal(moe(g, wu, wd, expert_bias=_negated(bias)), moe(g, wu, wd, expert_bias=bias))
    set_expert_gemm_precision("fp8")
    try:
        want = moe(g, wu.bfloat16(), wd.bfloat16())
        assert torch.equal(moe(g, _negated(wu), _negated(wd)), want)
    finally:
        set_expert_gemm_precision("bf16")

    gate, up, down = (torch.randn(*s, device=DEV).mul_(0.05).to(dtype) for s in ((256, 128), (256, 128), (128, 256)))
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        want = glu_ffn(x, gate, up, down, "swiglu")
        assert torch.equal(glu_ffn(_negated(x), _negated(gate), _negated(up), _negated(down), "swiglu"), want)

    def gate_gradient(of_loss):
        weight = g.detach().requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            losses = fused_moe(x, weight, wu, wd, top_k=2, gating="sigmoid", aux_loss_coeff=0.01, z_loss_coeff=0.01)[1]
        return torch.autograd.grad([losses["aux_loss"], losses["z_loss"]], weight, [of_loss, of_loss])[0]

    assert torch.equal(gate_gradient(_negated(torch.ones((), device=DEV))), gate_gradient(torch.ones((), device=DEV)))
