"""The order in which the grouped GEMM walks its tiles: experts in bands of units, at the heights where the number of bands
changes. A tile that the order left out or took twice would be missing from the result or belong to another place."""

import pytest
import torch

pytestmark = pytest.mark.gpu

from flashfusedmoe_b200 import _lib, ops  # noqa: E402

DEV = "cuda"


def _close(got, ref):
    # bf16 result of an fp32-accumulated product against fp64: 2^-9 relative from the rounding; the accumulation of K terms
    # of magnitude about 1 adds at most 2^-24 K sqrt(K) absolute, below 1e-3 for K <= 448
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-3).all()


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("units", [1, 11, 12, 13, 19, 20, 21, 28])
def test_grouped_rows(units, pair):
    """Two experts, the first `units` 256-row units high with a ragged end, times 1 and 3 column blocks."""
    g = torch.Generator(device=DEV).manual_seed(units)
    rows = [256 * units - 37, 300]
    starts = [0, 2 * units, 2 * units + 4]
    ts = torch.tensor(starts, dtype=torch.int32, device=DEV)
    cap, K = starts[-1] * 128, 128
    A = torch.randn(cap, K, generator=g, device=DEV).bfloat16()
    old = _lib.load().ffm_set_gemm_cta_pair(pair)
    try:
        for n_out in (64, 704):
            B = torch.randn(2, n_out, K, generator=g, device=DEV).bfloat16()
            got = ops.grouped_gemm(A, B.view(-1, K), _lib.B_KMAJOR, 2, ts, K, n_out)
            ops.check_status()
            for e, r in enumerate(rows):
                at = starts[e] * 128
                _close(got[at:at + r], A[at:at + r].double() @ B[e].double().T)
    finally:
        _lib.load().ffm_set_gemm_cta_pair(old)


@pytest.mark.parametrize("M,Nout", [(2816, 64), (3072, 320), (3136, 1088), (5184, 64), (7168, 320)])
def test_weight_gradient(M, Nout):
    """Two experts' gradients of 11 to 28 units by 1 to 5 column blocks, sums over a ragged and an ordinary number of rows."""
    g = torch.Generator(device=DEV).manual_seed(M + Nout)
    counts, starts = [133, 64], [0, 2, 4]
    A = torch.zeros(512, M, device=DEV).bfloat16()
    B = torch.zeros(512, Nout, device=DEV).bfloat16()
    for e, r in enumerate(counts):
        at = starts[e] * 128
        A[at:at + r] = torch.randn(r, M, generator=g, device=DEV).bfloat16()
        B[at:at + r] = torch.randn(r, Nout, generator=g, device=DEV).bfloat16()
    got = ops.grouped_gemm_wgrad(A, B, 2, torch.tensor(starts, dtype=torch.int32, device=DEV),
                                 counts=torch.tensor(counts, dtype=torch.int32, device=DEV))
    ops.check_status()
    for e, r in enumerate(counts):
        rows = slice(starts[e] * 128, starts[e] * 128 + r)
        _close(got[e], A[rows].double().T @ B[rows].double())


def _close_deep(got, ref, K):
    # as above; the accumulation of K terms, twice 2^-24 K sqrt(K): 0.07 at K = 7168, where products that belong elsewhere are off
    # by about sqrt(K) = 85
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + max(1e-3, 2.0 ** -23 * K * K ** 0.5)).all()


# more column blocks (26) than units: one band while the expert's rows fit a third of L2, bands beyond (K > 6826 at 12 pairs)
@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("K", [128, 7168])
def test_grouped_rows_with_more_column_blocks_than_units(K, pair):
    g = torch.Generator(device=DEV).manual_seed(K)
    rows, starts, n_out = [256 * 12 - 37, 300], [0, 24, 28], 6464
    ts = torch.tensor(starts, dtype=torch.int32, device=DEV)
    A = torch.randn(starts[-1] * 128, K, generator=g, device=DEV).bfloat16()
    B = torch.randn(2, n_out, K, generator=g, device=DEV).bfloat16()
    old = _lib.load().ffm_set_gemm_cta_pair(pair)
    try:
        got = ops.grouped_gemm(A, B.view(-1, K), _lib.B_KMAJOR, 2, ts, K, n_out)
    finally:
        _lib.load().ffm_set_gemm_cta_pair(old)
    ops.check_status()
    for e, r in enumerate(rows):
        at = starts[e] * 128
        _close_deep(got[at:at + r], A[at:at + r].double() @ B[e].double().T, K)


# the same for 13 units of a weight gradient: bands beyond sums over 6300 rows
@pytest.mark.parametrize("rows", [133, 6363])
def test_weight_gradient_with_more_column_blocks_than_units(rows):
    g = torch.Generator(device=DEV).manual_seed(rows)
    M, n_out = 3136, 6464
    tiles = (rows + 255) // 256 * 2
    counts, starts = [rows, 64], [0, tiles, tiles + 2]
    A = torch.zeros(starts[-1] * 128, M, device=DEV).bfloat16()
    B = torch.zeros(starts[-1] * 128, n_out, device=DEV).bfloat16()
    for e, r in enumerate(counts):
        at = starts[e] * 128
        A[at:at + r] = torch.randn(r, M, generator=g, device=DEV).bfloat16()
        B[at:at + r] = torch.randn(r, n_out, generator=g, device=DEV).bfloat16()
    got = ops.grouped_gemm_wgrad(A, B, 2, torch.tensor(starts, dtype=torch.int32, device=DEV),
                                 counts=torch.tensor(counts, dtype=torch.int32, device=DEV))
    ops.check_status()
    for e, r in enumerate(counts):
        at = slice(starts[e] * 128, starts[e] * 128 + r)
        _close_deep(got[e], A[at].double().T @ B[at].double(), r)
