"""Decode-sized calls whose contractions are long: the layer, which runs them as decode GEMMs, against the 256-row tiles, on both
sides of the lines of the rule (64 and 128 tokens, K = 8192), with one chain and with the permute."""

import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import _lib, fused_moe, ops  # noqa: E402

layer_module = importlib.import_module("flashfusedmoe_b200.fused_moe")
DEV = "cuda"


@pytest.mark.parametrize("N,D,H,E,chain", [(1, 2368, 64, 8, True), (3, 4096, 192, 8, True), (64, 8256, 64, 4, True),
                                           (65, 8192, 64, 8, True), (65, 8256, 64, 8, False), (128, 2560, 2368, 8, False),
                                           (37, 2368, 4160, 8, False)])
def test_long_contractions(N, D, H, E, chain):
    k = 2
    gen = torch.Generator(device=DEV).manual_seed(N + D)
    x = torch.randn(N, D, generator=gen, device=DEV).bfloat16()
    g, wu, wd = (torch.randn(*s, generator=gen, device=DEV).mul_(0.02).bfloat16() for s in ((E, D), (E, 2 * H, D), (E, D, H)))
    bits = layer_module._few_rows(N, D, E, k, H, False, None, None)
    assert bool(bits & layer_module._FEW_DECODE_UP) == (N <= 64 or D <= 8192) and bits & layer_module._FEW_DECODE_DOWN
    assert bool(bits & layer_module._FEW_ONE_CHAIN) == chain
    with torch.no_grad():
        got = fused_moe(x, g, wu, wd, top_k=k)[0].float()
    r = ops.route_forward(x, g, k)
    Xg = ops.permute_rows(x, r.src, ops.rows_capacity(N * k, E), k)
    act, _ = ops.grouped_gemm_glu(Xg, wu, wu.view(-1, D)[H:], 2 * H, E, r.tile_start, D, H, "swiglu", want_preact=False)
    ref = ops.combine_forward(ops.grouped_gemm(act, wd, _lib.B_KMAJOR, E, r.tile_start, H, D), r.pos, r.topk_w, N, k).float()
    ops.check_status()
    # the same products, summed in fp32: where the order of a sum moves a value over a rounding boundary, a pre-activation,
    # an activation or a row of Y differs by one bf16 ulp (2^-8); three in turn at most
    assert ((got - ref).abs() <= 3 * 2.0 ** -8 * ref.abs().max()).all()
