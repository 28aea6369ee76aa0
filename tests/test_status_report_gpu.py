"""A device-side failure code raises at a later call of the layer, once, without the host waiting for the GPU."""

import pytest
import torch

pytestmark = pytest.mark.gpu

import flashfusedmoe_b200 as ffm  # noqa: E402
from flashfusedmoe_b200 import ops  # noqa: E402

DEV = torch.device("cuda", 0)


def _inputs():
    g = torch.Generator(device=DEV).manual_seed(0)
    h = torch.randn(8, 64, generator=g, device=DEV).bfloat16()
    return (h, *(torch.randn(*s, generator=g, device=DEV).bfloat16() for s in ((4, 64), (4, 128, 64), (4, 64, 64))))


def _call(inputs=None):
    return ffm.fused_moe(*(inputs or _inputs()), top_k=2)[0]


def test_failure_surfaces_at_a_later_call_once():
    want = _call()
    ops.check_status()
    ops.status_tensor(DEV).fill_(103)   # as a kernel whose bounded wait ran out leaves it
    _call()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="103.*earlier call"):
        _call()
    assert torch.equal(_call(), want)
    ops.check_status()


def test_check_status_takes_the_report():
    _call()
    ops.status_tensor(DEV).fill_(101)
    _call()
    with pytest.raises(RuntimeError, match="101"):
        ops.check_status()
    _call()
    torch.cuda.synchronize()
    _call()
    ops.check_status()


def test_captured_call_reports_at_replay():
    inputs = _inputs()
    _call(inputs)
    ops.check_status()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _call(inputs)
    graph.replay()
    torch.cuda.synchronize()
    _call()
    ops.status_tensor(DEV).fill_(102)
    graph.replay()
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="102"):
        _call()
    ops.check_status()


@pytest.mark.parametrize("first", ["layer", "poll"])
def test_both_channels_report_once(first):
    """The expert-parallel path's copy of the word and the layer's own report carry one failure: it raises once, whichever
    of the two is looked at first."""
    _call()
    ops.poll_status()
    torch.cuda.synchronize()
    ops.poll_status(enqueue=False)
    ops.check_status()
    ops.status_tensor(DEV).fill_(101)
    _call()               # the layer's last kernel stores the code
    ops.poll_status()     # and a copy of the word is queued
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="101.*earlier call"):
        _call() if first == "layer" else ops.poll_status()
    _call()
    ops.poll_status()
    torch.cuda.synchronize()
    _call()
    ops.poll_status()
    torch.cuda.synchronize()
    ops.poll_status(enqueue=False)
    ops.check_status()


def test_code_read_with_other_data_clears_both_channels():
    _call()
    ops.status_tensor(DEV).fill_(103)
    _call()
    ops.poll_status()
    with pytest.raises(RuntimeError, match="103"):
        ops.raise_on_status(103, DEV)
    torch.cuda.synchronize()
    _call()
    ops.poll_status(enqueue=False)
    ops.check_status()
