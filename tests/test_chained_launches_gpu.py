"""The launches of a call as one native call enqueues them: the layer's calls without a shared expert against the same kernels
launched one by one, at sizes of the routes through the bf16 forward pass and for calls queued without a pause."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import _lib, fused_moe, ops  # noqa: E402

DEV = "cuda"


def _one_by_one(x, g, wu, wd, k):
    N, D = x.shape
    E, H = wu.shape[0], wu.shape[1] // 2
    r = ops.route_forward(x, g, k)
    Xg = ops.permute_rows(x, r.src, ops.rows_capacity(N * k, E), k)
    act, _ = ops.grouped_gemm_glu(Xg, wu, wu.view(-1, D)[H:], 2 * H, E, r.tile_start, D, H, "swiglu", want_preact=False)
    Y = ops.grouped_gemm(act, wd, _lib.B_KMAJOR, E, r.tile_start, H, D)
    return ops.combine_forward(Y, r.pos, r.topk_w, N, k)


# one chain with gathered rows; decode GEMMs behind a permute (weights above one chain's bound are too large for a test: 129
# tokens take the 128-row tiles); 256-row tiles with two, and with many, launches of routing; 32 experts: gate GEMM
@pytest.mark.parametrize("E", [8, 32])
@pytest.mark.parametrize("N", [1, 64, 129, 300, 4001])
def test_layer_against_single_launches(N, E):
    """Bit for bit, 12 calls with other tokens each, queued without a pause."""
    D, H, k = 256, 512, 2
    gen = torch.Generator(device=DEV).manual_seed(N + E)
    g, wu, wd = (torch.randn(*s, generator=gen, device=DEV).mul_(0.05).bfloat16() for s in ((E, D), (E, 2 * H, D), (E, D, H)))
    xs = [torch.randn(N, D, generator=gen, device=DEV).bfloat16() for _ in range(12)]
    with torch.no_grad():
        want = [_one_by_one(x, g, wu, wd, k) for x in xs]
        torch.cuda.synchronize()
        got = [fused_moe(x, g, wu, wd, top_k=k)[0] for x in xs]
    ops.check_status()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
