"""Build libffmoe.so (sm_100a only, nvcc) and its torch side (g++; _lib.native_path) in-tree.

Usage: python -m flashfusedmoe_b200.build [--force]
The shared libraries land next to this file so that they travel with the source tree.
"""

import os
import shutil
import subprocess
import sys
import sysconfig

from ._lib import native_path

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libffmoe.so")
NATIVE_SOURCE = os.path.join(CSRC, "ffm_torch.cpp")
PTXAS_LOG = os.path.join(HERE, "libffmoe.ptxas.txt")
SOURCES = ["ffm_api.cu", "ffm_route.cu", "ffm_rows.cu", "ffm_route_bwd.cu", "ffm_gemm_sm100.cu", "ffm_gemm_tok_sm100.cu",
           "ffm_p2p.cu", "ffm_fp8.cu", "ffm_layer.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--use_fast_math", "-Xptxas", "-v",
]


def _newest_source_mtime():
    paths = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith(".o")]
    paths.append(os.path.join(HERE, "..", "include", "ffmoe.h"))
    return max(os.path.getmtime(p) for p in paths)


def _native_command(target):
    """g++ command of the torch extension: host code only, against the installed torch's headers and libraries."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_EXTENSION_NAME=_native",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + ["-I" + d for d in include] +
            [NATIVE_SOURCE, "-o", target, "-L" + os.path.join(root, "lib"), "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10"])


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ into libffmoe.so and ffm_torch.cpp into the torch extension. Returns the first one's path."""
    newest, native = _newest_source_mtime(), native_path()
    if not force and all(os.path.exists(f) and os.path.getmtime(f) >= newest for f in (LIB, native)):
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    objs = []
    procs = [("ffm_torch.cpp", subprocess.Popen(_native_command(native), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                                text=True))]
    for src in SOURCES:
        obj = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc] + NVCC_FLAGS + ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    log = []
    for src, p in procs:
        out, _ = p.communicate()
        log.append(out)
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"compiling {src} failed")
    # ptxas -v output (registers, spills, shared memory per kernel), kept beside the library: the GLU-epilogue GEMM
    # is sensitive to register allocation (tests/test_cabi_cpu.py checks it)
    with open(PTXAS_LOG, "w") as f:
        f.write("".join(log))
    cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-lcudart"]
    subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
