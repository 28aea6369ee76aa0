"""GEMMs of decode-sized calls and weight gradients that end at the last valid row, against torch in fp32, at the edges of
their tiles: 8- and 16-row boxes, the 64-token tile, several token tiles per expert, features that do not fill a tile,
empty experts.

Bounds: products of bf16 values are exact in fp32, so an output differs from the fp32 evaluation by its own rounding to
bf16 (2^-9 relative) and the order of the sum (below 1e-5 of the sum of magnitudes at these K)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import ops  # noqa: E402
from test_kernels_gpu import glu_ref  # noqa: E402

DEV = "cuda"
COUNTS = [5, 0, 200, 128, 31, 32, 33, 256, 257, 300, 1, 15, 16, 17, 64, 65, 600]
SENTINEL = -7.0


def layout(counts):
    """tile_start, counts, first rows and the row count of the 256-row-aligned grouped layout."""
    base, starts, tiles = 0, [], [0]
    for c in counts:
        starts.append(base)
        base += (c + 255) // 256 * 256
        tiles.append(base // 128)
    i32 = dict(dtype=torch.int32, device=DEV)
    return torch.tensor(tiles, **i32), torch.tensor(counts, **i32), starts, base


def grouped(counts, starts, rows, width, g, box=1):
    """Random valid rows, zeros up to the next multiple of `box`, NaN beyond."""
    x = torch.full((rows, width), float("nan"), device=DEV).bfloat16()
    for c, s in zip(counts, starts):
        x[s:s + (c + box - 1) // box * box] = 0
        x[s:s + c] = torch.randn(c, width, generator=g, device=DEV).bfloat16()
    return x


def check(got, ref, mag):
    got, ref = got.float(), ref.float()
    assert torch.isfinite(got).all()
    assert ((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * mag).all()


def check_glu(act, pre32, H, activation, mag):
    """`act` against the activation of the bf16-rounded pre-activations; a pre-activation within 1e-5 of its sum of
    magnitudes of a rounding boundary may round to the neighbour (one part in 2^8)."""
    pre = pre32.bfloat16().float()
    ref = glu_ref(activation, pre[:, :H], pre[:, H:]).float()
    near = ((pre32 - pre).abs() >= pre.abs() * 2.0 ** -9 * 0.9 - 1e-5 * mag)
    near = near[:, :H] | near[:, H:]
    err = (act.float() - ref).abs()
    up = pre[:, H:].abs()
    assert torch.isfinite(act.float()).all()
    assert (err <= 2.0 ** -8 * ref.abs() + 1e-4 * up)[~near].all()
    assert (err <= 2.0 ** -5 * (ref.abs() + up * (1 + pre[:, :H].abs())) + 1e-4)[near].all()


def with_sentinel(monkeypatch, fn):
    """fn() with its bf16 outputs allocated full of a sentinel, so that rows nothing may touch can be told."""
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **k: empty(*a, **k).fill_(SENTINEL) if k.get("dtype") ==
                        torch.bfloat16 else empty(*a, **k))
    out = fn()
    monkeypatch.undo()
    ops.check_status()
    return out


def untouched(out, starts):
    for c, s in zip(COUNTS, starts):
        assert (out[s + (c + 7) // 8 * 8:s + (c + 255) // 256 * 256] == SENTINEL).all()


def valid(starts):
    return [(e, slice(s, s + c)) for e, (c, s) in enumerate(zip(COUNTS, starts)) if c]


@pytest.mark.parametrize("K,Nout", [(64, 32), (192, 128), (128, 288), (1024, 320)])
def test_decode_gemm(K, Nout, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(K + Nout)
    ts, cn, starts, rows = layout(COUNTS)
    x = grouped(COUNTS, starts, rows, K, g)
    w = torch.randn(len(COUNTS), Nout, K, generator=g, device=DEV).bfloat16()
    out = with_sentinel(monkeypatch, lambda: ops.decode_gemm(x, w, len(COUNTS), ts, cn, K, Nout))
    for e, r in valid(starts):
        check(out[r], x[r].float() @ w[e].float().T, x[r].float().abs() @ w[e].float().abs().T)
    untouched(out, starts)


@pytest.mark.parametrize("activation", ["swiglu", "geglu", "relu_squared", "geglu_erf"])
@pytest.mark.parametrize("K,H", [(64, 64), (192, 128), (576, 320)])
def test_decode_gemm_glu(K, H, activation, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(K + H)
    ts, cn, starts, rows = layout(COUNTS)
    x = grouped(COUNTS, starts, rows, K, g)
    w = (torch.randn(len(COUNTS), 2 * H, K, generator=g, device=DEV) * 0.2).bfloat16()
    act = with_sentinel(monkeypatch, lambda: ops.decode_gemm_glu(x, w, w.view(-1, K)[H:], 2 * H, len(COUNTS), ts, cn, K,
                                                                 H, activation))
    for e, r in valid(starts):
        check_glu(act[r], x[r].float() @ w[e].float().T, H, activation, x[r].float().abs() @ w[e].float().abs().T)
    untouched(act, starts)


@pytest.mark.parametrize("rows", [1, 8, 33, 64, 100])
@pytest.mark.parametrize("swap", [False, True])
def test_dense(rows, swap):
    """The shared expert: separate gate and up tensors in either address order, row counts that are no multiple of 8."""
    g = torch.Generator(device=DEV).manual_seed(rows)
    K, H = 128, 192
    pair = (torch.randn(2, H, K, generator=g, device=DEV) * 0.2).bfloat16()
    wg, wu = (pair[1], pair[0]) if swap else (pair[0], pair[1])
    x = torch.randn(rows, K, generator=g, device=DEV).bfloat16()
    act = ops.decode_gemm_glu(x, wg, wu, H, 1, None, None, K, H, "swiglu")
    both = torch.cat([wg, wu]).float()
    check_glu(act, x.float() @ both.T, H, "swiglu", x.float().abs() @ both.abs().T)
    w = torch.randn(K, H, generator=g, device=DEV).bfloat16()
    out = ops.decode_gemm(act, w, 1, None, None, H, K)
    ops.check_status()
    check(out, act.float() @ w.float().T, act.float().abs() @ w.float().abs().T)


@pytest.mark.parametrize("M,Nout", [(64, 64), (192, 320)])
def test_wgrad_up_to_the_last_valid_row(M, Nout):
    """Bit for bit the sum over the whole zero-padded segments; what lies past the next multiple of 16 is not read."""
    g = torch.Generator(device=DEV).manual_seed(M)
    ts, cn, starts, rows = layout(COUNTS)
    a, b = grouped(COUNTS, starts, rows, M, g, box=16), grouped(COUNTS, starts, rows, Nout, g, box=16)
    got = ops.grouped_gemm_wgrad(a, b, len(COUNTS), ts, counts=cn)
    ref = ops.grouped_gemm_wgrad(torch.nan_to_num(a), torch.nan_to_num(b), len(COUNTS), ts)
    ops.check_status()
    assert torch.equal(got, ref)
