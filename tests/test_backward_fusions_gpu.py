"""Backward-pass kernels that take over separate launches: two addends in the combine, a contraction over two weight
tensors, and the routing term of the input gradient as a GEMM when every logit has a gradient."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import _lib, ops  # noqa: E402

DEV = "cuda"


@pytest.mark.parametrize("N,D,k", [(1, 8, 1), (33, 264, 3), (100, 2048, 4), (257, 72, 5), (64, 1024, 8)])
def test_combine_with_two_addends(N, D, k):
    """Bit for bit the combine, then one bf16 addition per addend."""
    g = torch.Generator(device=DEV).manual_seed(N + D)
    Y = torch.randn(N * k + 7, D, generator=g, device=DEV).bfloat16()
    pos = torch.randperm(N * k + 7, generator=g, device=DEV)[:N * k].int()
    w = torch.rand(N, k, generator=g, device=DEV)
    a, b = (torch.randn(N, D, generator=g, device=DEV).bfloat16() for _ in range(2))
    plain = ops.combine_forward(Y, pos, w, N, k)
    assert torch.equal(ops.combine_forward(Y, pos, w, N, k, addend=a, addend2=b), plain + a + b)
    assert torch.equal(ops.combine_forward(Y, pos, w, N, k, addend2=b), plain + b)
    ref = (Y[pos.long()].view(N, k, D).float() * w.bfloat16().float().unsqueeze(-1)).sum(1)
    # rounding to bf16, and k fp32 additions in another order
    assert ((plain.float() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()


@pytest.mark.parametrize("rows,K1,K2,Nout", [(1, 64, 64, 64), (130, 64, 192, 320), (2000, 1024, 448, 128)])
def test_dense_gemm_two(rows, K1, K2, Nout):
    """Bit for bit the GEMM on the concatenated weights."""
    g = torch.Generator(device=DEV).manual_seed(rows)
    A = torch.randn(rows, K1 + K2, generator=g, device=DEV).bfloat16()
    B = torch.randn(K1 + K2, Nout, generator=g, device=DEV).bfloat16()
    got = ops.dense_gemm_two(A, B[:K1].clone(), B[K1:].clone())
    ref = ops.grouped_gemm(A, B, _lib.B_NMAJOR, 1, None, K1 + K2, Nout)
    ops.check_status()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("gating,loss", [("softmax", "z"), ("sigmoid", "aux"), ("sigmoid", "both")])
@pytest.mark.parametrize("N,D,E,k", [(1, 64, 64, 2), (129, 192, 64, 6), (300, 128, 192, 8), (77, 64, 16, 3)])
def test_dense_logit_gradient(N, D, E, k, gating, loss):
    """dH and dGate of a loss whose gradient reaches every logit, against autograd in fp64 on the same choice. Every
    gradient of a logit is rounded to bf16 (2^-9 relative), and so is the result."""
    g = torch.Generator(device=DEV).manual_seed(N + E)
    hidden = torch.randn(N, D, generator=g, device=DEV).bfloat16()
    gate = (torch.randn(E, D, generator=g, device=DEV) * 0.2).bfloat16()
    r = ops.route_forward(hidden, gate, k, gating)
    gw = torch.randn(N * k, generator=g, device=DEV)
    gaux = torch.rand(E, generator=g, device=DEV) * N if loss != "z" else None
    gz = torch.full((1,), 0.7, device=DEV) if loss != "aux" else None
    dH, dG = ops.route_backward(gw, r, gaux, gz, hidden, gate, gating)
    ops.check_status()
    lg = r.logits.double().requires_grad_()
    val = lg if gating == "softmax" else torch.sigmoid(lg)
    p = val.gather(1, r.topk_idx.long())
    w = torch.softmax(p, 1) if gating == "softmax" else p / (p.sum(1, keepdim=True) + 1e-6)
    obj = (w.reshape(-1) * gw.double()).sum()
    if gaux is not None:
        obj = obj + (torch.sigmoid(lg).mean(0) * gaux.double()).sum()
    if gz is not None:
        obj = obj + 0.7 * torch.logsumexp(lg, 1).square().mean()
    gl = torch.autograd.grad(obj, lg)[0]
    for got, ref, mag in ((dH, gl @ gate.double(), gl.abs() @ gate.double().abs()),
                          (dG, gl.T @ hidden.double(), gl.abs().T @ hidden.double().abs())):
        assert ((got.double() - ref).abs() <= 2.0 ** -8 * (ref.abs() + mag) + 1e-5 * mag).all()
