"""GEMMs of decode-sized calls and weight gradients that end at the last valid row, against torch in fp32, at the edges of
their tiles: 4-, 8- and 16-row boxes, the 64-token tile, several token tiles per expert, features that do not fill a tile,
empty experts.

Bounds: products of bf16 values are exact in fp32, so an output differs from the fp32 evaluation by its own rounding to
bf16 (2^-9 relative) and the order of the sum (below 1e-5 of the sum of magnitudes at these K)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import _lib, ops  # noqa: E402
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


@pytest.mark.parametrize("H,D", [(64, 32), (192, 128), (128, 288), (1024, 320)])
def test_decode_down(H, D, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(H + D)
    ts, cn, starts, rows = layout(COUNTS)
    N, k = sum(COUNTS), 1
    x = grouped(COUNTS, starts, rows, H, g)
    w = torch.randn(len(COUNTS), D, H, generator=g, device=DEV).bfloat16()
    out, none = with_sentinel(monkeypatch, lambda: ops.decode_down(x, ts, cn, k, N, w))
    assert none is None
    for e, r in valid(starts):
        check(out[r], x[r].float() @ w[e].float().T, x[r].float().abs() @ w[e].float().abs().T)
    untouched(out, starts)


@pytest.mark.parametrize("activation", ["swiglu", "geglu", "relu_squared", "geglu_erf"])
@pytest.mark.parametrize("D,H,k", [(64, 64, 1), (192, 128, 3), (576, 320, 2)])
def test_decode_up(D, H, k, activation, monkeypatch):
    """Token rows gathered through src, every token in several experts."""
    g = torch.Generator(device=DEV).manual_seed(D + H)
    ts, cn, starts, rows = layout(COUNTS)
    T = sum(COUNTS)
    N = -(-T // k)
    slots = torch.randperm(N * k, generator=g, device=DEV)[:T].int()
    src = torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    at = 0
    for c, s in zip(COUNTS, starts):
        src[s:s + c] = slots[at:at + c]
        at += c
    hidden = torch.randn(N, D, generator=g, device=DEV).bfloat16()
    w = (torch.randn(len(COUNTS), 2 * H, D, generator=g, device=DEV) * 0.2).bfloat16()
    act, none = with_sentinel(monkeypatch, lambda: ops.decode_up(hidden, src, k, ts, cn, rows, w, activation))
    assert none is None
    for e, r in valid(starts):
        x = hidden[(src[r] // k).long()].float()
        check_glu(act[r], x @ w[e].float().T, H, activation, x.abs() @ w[e].float().abs().T)
    untouched(act, starts)
    rows_grouped = torch.full((rows, D), float("nan"), device=DEV).bfloat16()
    for _, r in valid(starts):
        rows_grouped[r] = hidden[(src[r] // k).long()]
    same, _ = ops.decode_up(rows_grouped, None, k, ts, cn, rows, w, activation)
    ops.check_status()
    for _, r in valid(starts):
        assert torch.equal(same[r], act[r])


@pytest.mark.parametrize("N", [1, 3, 17, 64, 100])
@pytest.mark.parametrize("swap", [False, True])
def test_shared_expert_inside(N, swap):
    """Separate gate and up tensors in either address order, other widths than the routed experts, row counts that are no
    multiple of 8; the routed outputs are those of a launch without it."""
    g = torch.Generator(device=DEV).manual_seed(N)
    D, H, Hs, E, k = 128, 64, 192, 5, 2
    hidden = torch.randn(N, D, generator=g, device=DEV).bfloat16()
    r = ops.route_forward(hidden, torch.randn(E, D, generator=g, device=DEV).bfloat16(), k)
    wu = (torch.randn(E, 2 * H, D, generator=g, device=DEV) * 0.2).bfloat16()
    wd = torch.randn(E, D, H, generator=g, device=DEV).bfloat16()
    pair = (torch.randn(2, Hs, D, generator=g, device=DEV) * 0.2).bfloat16()
    wg, wup = (pair[1], pair[0]) if swap else (pair[0], pair[1])
    sd = torch.randn(D, Hs, generator=g, device=DEV).bfloat16()
    act, s_act = ops.decode_up(hidden, r.src, k, r.tile_start, r.counts, r.rows_cap, wu, "swiglu",
                               (hidden, wg, wup, "geglu_erf"))
    alone, _ = ops.decode_up(hidden, r.src, k, r.tile_start, r.counts, r.rows_cap, wu, "swiglu")
    Y, s_out = ops.decode_down(act, r.tile_start, r.counts, k, N, wd, (s_act, sd))
    Y1, _ = ops.decode_down(act, r.tile_start, r.counts, k, N, wd)
    _, s_alone = ops.decode_up(None, None, k, None, None, 0, None, "swiglu", (hidden, wg, wup, "geglu_erf"))
    _, o_alone = ops.decode_down(None, None, None, k, N, None, (s_act, sd))
    assert torch.equal(s_alone, s_act) and torch.equal(o_alone, s_out)
    ops.check_status()
    rows = r.pos.long()
    assert torch.equal(act[rows], alone[rows]) and torch.equal(Y[rows], Y1[rows])
    both = torch.cat([wg, wup]).float()
    check_glu(s_act, hidden.float() @ both.T, Hs, "geglu_erf", hidden.float().abs() @ both.abs().T)
    check(s_out, s_act.float() @ sd.float().T, s_act.float().abs() @ sd.float().abs().T)


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


def test_a_wait_that_runs_out_ends_the_launch():
    """With the shortest wait a CTA may give up: it reports that, takes its copies and MMAs in flight along, and the next
    launch is right."""
    torch.manual_seed(0)
    x = torch.randn(64, 2048, device=DEV).bfloat16()
    gate, up = (torch.randn(2816, 2048, device=DEV).bfloat16() for _ in range(2))
    shared = (x, gate, up, "swiglu")
    want = ops.decode_up(None, None, 1, None, None, 0, None, "swiglu", shared=shared)[1]
    ops.check_status()
    lib = _lib.load()
    old = lib.ffm_set_wait_cycles(1)
    try:
        for _ in range(3):
            ops.decode_up(None, None, 1, None, None, 0, None, "swiglu", shared=shared)
        torch.cuda.synchronize()
    finally:
        lib.ffm_set_wait_cycles(old)
    assert int(ops.status_tensor(x.device).item()) in (0, 101, 102, 103)
    ops.status_tensor(x.device).zero_()
    assert torch.equal(ops.decode_up(None, None, 1, None, None, 0, None, "swiglu", shared=shared)[1], want)
    ops.check_status()
