"""CPU: what the library's host side finds out once per device is not carried from one device to another. The launch code's
own helper is compiled against a stand-in for cudaGetDevice."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "ffm_device.h"
#include <cstdio>
static int current = 0;
static bool broken = false;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = current; return broken ? cudaErrorUnknown : cudaSuccess; }
int main() {
  static ffm::PerDevice v;
  int calls = 0;
  auto on = [&](int dev, int found) { current = dev; return v.get([&] { ++calls; return found; }); };
  bool ok = on(0, 5) == 5 && on(0, 6) == 5 && calls == 1;   // found once
  ok = ok && on(1, 7) == 7 && on(0, 0) == 5 && on(1, 0) == 7 && calls == 2;   // per device
  ok = ok && on(2, 0) == 0 && on(2, 3) == 3 && calls == 4;   // a failure is tried again
  ok = ok && on(1000, 9) == 9 && on(-1, 8) == 8 && calls == 6;   // no slot: asked every time
  broken = true;
  ok = ok && on(0, 4) == 4 && calls == 7;
  return ok ? 0 : 1;
}
"""


def test_values_belong_to_a_device(tmp_path):
    source, program = tmp_path / "t.cpp", tmp_path / "t"
    source.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT}/flashfusedmoe_b200/csrc", f"-I{cuda}/include", str(source),
                    "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0


def test_launch_code_keeps_nothing_for_the_process():
    """Every cudaFuncSetAttribute of the library stands inside a per-device value."""
    csrc = os.path.join(ROOT, "flashfusedmoe_b200", "csrc")
    found = 0
    for name in sorted(os.listdir(csrc)):
        if not name.endswith((".cu", ".cuh")):
            continue
        lines = open(os.path.join(csrc, name)).read().splitlines()
        for i, line in enumerate(lines):
            if "cudaFuncSetAttribute(" in line:
                found += 1
                assert any(".get([&]" in before for before in lines[max(0, i - 3):i]), f"{name}:{i + 1}"
    assert found >= 3
