"""CPU: libffmoe.so loads, exports every symbol include/ffmoe.h declares, and its host-only entry points
answer without a GPU. No compute kernel is launched here."""

import ctypes
import inspect
import multiprocessing
import os
import re

import pytest

from flashfusedmoe_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "ffmoe.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(ffm_[a-z_0-9]+)\s*\(", text)))


def test_library_is_built():
    assert os.path.exists(_lib.LIB_PATH), "run `python -m flashfusedmoe_b200.build` first"


def test_every_declared_symbol_is_exported_and_bound():
    lib = ctypes.CDLL(_lib.LIB_PATH)
    names = declared_symbols()
    assert len(names) >= 16
    for name in names:
        assert hasattr(lib, name), f"{name} declared in ffmoe.h but not exported"
        assert name in _lib.SIGNATURES, f"{name} has no ctypes prototype in _lib.SIGNATURES"
    assert sorted(_lib.SIGNATURES) == names


def test_host_only_entry_points():
    lib = _lib.load()
    assert lib.ffm_version() == 100
    assert _lib.error_string(0) == "ok"
    assert "workspace" in _lib.error_string(-4)
    assert "epilogue" in _lib.error_string(103)
    # rows capacity: 256 * floor((T + 255 E) / 256)
    assert lib.ffm_rows_capacity(32768, 8) == 256 * ((32768 + 255 * 8) // 256)
    assert lib.ffm_rows_capacity(0, 4) == 256 * ((255 * 4) // 256)
    assert lib.ffm_set_gemm_cta_pair(-1) in (0, 1)
    assert lib.ffm_route_workspace_bytes(16384, 8, 2) > 0
    assert lib.ffm_route_backward_workspace_bytes(16384, 1024, 8) > 16384 * 8 * 2
    old = lib.ffm_set_wait_cycles(12345)
    assert lib.ffm_set_wait_cycles(old) == 12345


def test_argument_validation_without_gpu():
    lib = _lib.load()
    # null pointers are rejected before any CUDA call
    assert lib.ffm_permute_rows(0, 0, 128, 1, 64, 1, 0, 0) == -1
    assert lib.ffm_grouped_gemm(0, 0, 0, 1, 0, 128, 64, 64, 1.0, 0, 0, 0, 0, 0) == -1
    assert lib.ffm_combine_forward(0, 0, 0, 0, 4, 2, 64, 0, 0) == -1


def test_groups_too_small_for_top_k_are_refused():
    """A token cannot choose top_k experts from fewer: refused before any CUDA call (the workspace check comes after)."""
    lib = _lib.load()

    def route(topk_group, top_k):
        E, N, D = 8, 4, 64
        return lib.ffm_route_forward(1, 1, 0, N, D, E, top_k, 0, 1.0, 0, 4, topk_group, 1, 1, 1, 1, 1, 1, 1, 1,
                                     lib.ffm_rows_capacity(N * top_k, E), 1, 1, 0, 1, 0)

    assert route(1, 3) == -1 and route(2, 5) == -1
    assert route(1, 2) == -4 and route(2, 4) == -4


def _check_operand_addresses():
    """Each operand in turn off its boundary; with fitting addresses a call gets as far as its launch, which fails without a device."""
    lib = _lib.load()
    a, off = 256, 260
    N, D, E, k = 512, 64, 8, 2
    cap, big = lib.ffm_rows_capacity(N * k, E), 1 << 30
    for call in (
            lambda hidden, gate: lib.ffm_route_forward(hidden, gate, 0, N, D, E, k, 0, 1.0, 0, 0, 0, a, a, a, a, a, a, a, a, cap, a,
                                                       a, big, a, 0),
            lambda hidden, gate, dH, workspace: lib.ffm_route_backward(a, a, a, a, a, 0, 0, hidden, gate, N, D, E, k, 0, 0, dH, a,
                                                                       workspace, big, a, 0),
            lambda x, grouped: lib.ffm_permute_rows(x, a, cap, k, D, 1, grouped, 0),
            lambda Y, add, add2, out: lib.ffm_combine_forward_add2(Y, a, a, add, add2, N, k, D, out, 0),
            lambda go, Y, gYw: lib.ffm_combine_backward(go, Y, a, a, cap, k, D, gYw, a, 0),
            lambda d_act, preact, gU: lib.ffm_glu_backward(d_act, preact, a, E, cap, D, 0, gU, 0),
            lambda x, q: lib.ffm_quantize_rows_e4m3(x, cap, D, q, a, 0),
            lambda x, q: lib.ffm_quantize_rows_given_scale_e4m3(x, cap, D, 128, a, q, 0),
            lambda d_act, preact, gU: lib.ffm_grouped_gemm_wgrad_glu_backward(a, a, E, a, cap, D, D, 1.0, a, d_act, preact, cap, D, 0,
                                                                              gU, a, 0)):
        names = inspect.signature(call).parameters
        fitting = dict.fromkeys(names, a)
        assert call(**fitting) not in (0, -1, -2)
        for name in names:
            assert call(**{**fitting, name: off}) == -2, (inspect.getsource(call), name)


def test_operands_off_a_16_byte_boundary_are_refused(monkeypatch):
    """Kernels that load and store 16 bytes at a time would end the context on such an address. In a process that sees no device."""
    monkeypatch.setenv("CUDA_VISIBLE_DEVICES", "")
    child = multiprocessing.get_context("spawn").Process(target=_check_operand_addresses)
    child.start()
    child.join()
    assert child.exitcode == 0


def _block_fields(name):
    """(field, "q" or "d") in the order in which include/ffmoe.h declares the fields of an argument block."""
    text = open(os.path.join(ROOT, "include", "ffmoe.h")).read()
    body = re.sub(r"/\*.*?\*/", "", text, flags=re.S).split("} " + name + ";")[0].rsplit("typedef struct {", 1)[1]
    fields = []
    for line in body.split(";"):
        line = line.replace("const", " ").strip()
        if line:
            kind, names = line.split(None, 1)
            for n in names.split(","):
                value = n.strip()
                assert kind in ("int64_t", "double") or value.startswith("*") or kind == "ffm_stream_t", (kind, value)
                fields.append((value.lstrip("*"), "d" if kind == "double" and not value.startswith("*") else "q"))
    return fields


@pytest.mark.parametrize("name,backward", [("ffm_layer_forward_args", 0), ("ffm_layer_backward_args", 1)])
def test_argument_block_is_packed_as_declared(name, backward):
    """Eight bytes a field: the packing, the header and the compiled struct agree in number, kinds and size."""
    from flashfusedmoe_b200 import ops
    packing = ops.LAYER_BACKWARD_ARGS if backward else ops.LAYER_FORWARD_ARGS
    fields = _block_fields(name)
    assert [n for n, _ in fields[-2:]] == ["timer", "launched"]
    packed = "".join(c * int(n) for n, c in re.findall(r"(\d+)([qd])", packing.format))
    assert packed == "".join(k for _, k in fields[:-2])
    assert _lib.load().ffm_layer_args_bytes(backward) == 8 * len(fields) == packing.size + 16


def test_layer_forward_refuses_launches_that_read_unwritten_buffers():
    """Every other field is zero: a combination that is let through fails on its null pointers, at another site."""
    from flashfusedmoe_b200 import ops
    lib = _lib.load()
    names = [n for n, _ in _block_fields("ffm_layer_forward_args")]

    def site(**values):
        fields = dict.fromkeys(names, 0)
        fields.update(dict(N=4, D=64, E=8, top_k=2, H=64, rows_cap=2048, capacity=-1), **values)
        launched = (ctypes.c_int64 * 3)()
        block = ops.LAYER_FORWARD_ARGS.pack(*[fields[n] for n in names[:-2]])
        rc = lib.ffm_layer_forward(block + (0).to_bytes(8, "little") + ctypes.addressof(launched).to_bytes(8, "little"))
        assert rc == -1
        return launched[2]

    tiles, up, down, shared, chain = 1, 2, 4, 8, 16
    refused, route, shared_up = 6, 2, 0
    for few in (chain, tiles | chain, up | chain, tiles | up | chain, down | chain, 32):
        assert site(few_rows=few) == refused
    assert site(few_rows=up | down | chain, capacity=4) == refused
    assert site(few_rows=up | down | chain, Hs=64) == refused
    for few in (up, down, shared):
        assert site(few_rows=few, need_grad=1) == refused
        assert site(few_rows=few, preact=16) == refused
    assert site(few_rows=up, fp8=1) == refused
    for few in (0, tiles, tiles | up, tiles | down, tiles | up | down, tiles | up | down | chain):
        assert site(few_rows=few) == route
    assert site(few_rows=tiles | up | down | shared | chain, Hs=64) == route
    assert site(few_rows=shared, Hs=64) == shared_up


def test_no_kernel_is_launched_ahead_of_the_one_before_it():
    """Programmatic stream serialization is ordered with the kernel right before on the stream, and this library does not know
    what that is: another thread's event, or the allocator's, may lie between two launches of a call. Kernels here also read
    what the one before wrote through the read-only path, which holds only if that kernel has ended."""
    csrc = os.path.join(os.path.dirname(_lib.LIB_PATH), "csrc")
    for name in sorted(os.listdir(csrc)):
        if name.endswith((".cu", ".cuh", ".h", ".cpp")):
            text = open(os.path.join(csrc, name)).read()
            assert not re.search(r"griddepcontrol|cudaGridDependency|cudaTriggerProgrammatic|LaunchAttributeProgrammatic", text), name


def test_extension_of_another_torch_is_built_again(monkeypatch):
    """The torch extension belongs to one torch and one Python: after a change build() compiles, and nothing loads the old file."""
    import torch
    from flashfusedmoe_b200 import build

    class Compiled(Exception):
        pass

    def compiler(*args, **kwargs):
        raise Compiled

    assert build.build(force=False) == build.LIB
    monkeypatch.setattr(build.subprocess, "Popen", compiler)
    assert build.build(force=False) == build.LIB
    monkeypatch.setattr(_lib, "_native", None)
    monkeypatch.setattr(torch, "__version__", "0.0.0+other")
    with pytest.raises(Compiled):
        build.build(force=False)
    with pytest.raises(RuntimeError, match="not built for this torch.*flashfusedmoe_b200.build"):
        _lib.native()
    monkeypatch.undo()
    monkeypatch.setattr(build.subprocess, "Popen", compiler)
    monkeypatch.setattr(build.sysconfig, "get_config_var", lambda name: ".cpython-399-x86_64-linux-gnu.so")
    with pytest.raises(Compiled):
        build.build(force=False)


def test_product_path_has_no_cpu_fallback():
    import torch
    from flashfusedmoe_b200 import fused_moe
    h = torch.randn(4, 64).bfloat16()
    g = torch.randn(4, 64).bfloat16()
    wu = torch.randn(4, 128, 64).bfloat16()
    wd = torch.randn(4, 64, 64).bfloat16()
    with pytest.raises(RuntimeError, match="no CPU path"):
        fused_moe(h, g, wu, wd, top_k=2)


def test_gemm_register_allocation_canary():
    """ptxas figures of the build: no GEMM instantiation spills, and the instantiations with helper epilogue warps
    (320 threads: both GLU epilogues) stay far below the 204 registers that thread count allows. (The first GLU
    epilogue kept 128 accumulator values in flight per lane, needed 234 registers, and ran 30 % slower when an unrelated
    change to the parameter struct made ptxas pick 185; the rolled epilogues hold 32.)"""
    import re
    from flashfusedmoe_b200 import build
    build.build(force=not os.path.exists(build.PTXAS_LOG))
    text = open(build.PTXAS_LOG).read()
    blocks = re.findall(r"Compiling entry function '(\S*ffm_gemm_kernel\S*)'.*?Used (\d+) registers", text, flags=re.S)
    assert len(blocks) >= 10, "ptxas output of the GEMM instantiations not found"
    spills = re.findall(r"ffm_gemm_kernel\S*\n\s*(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", text)
    assert spills and all(int(a) == 0 and int(b) == 0 for _, a, b in spills), "a GEMM instantiation spills registers"
    # <A, B, EPI_GLU = 1 or EPI_GLUBWD = 2, ...>
    glu = [int(r) for name, r in blocks if re.search(r"ILi\dELi\dELi[12]ELi", name)]
    assert glu and max(glu) <= 160, f"GLU-epilogue GEMM register allocation changed: {glu}"
