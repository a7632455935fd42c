"""The contraction's shared-memory opt-in holds for one device: it is made on each
device a process contracts on (csrc/once_per_device.h, on the host alone; this
suite's machines have one GPU)."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "monte-carlo-simulation-3d-rms_b200", "csrc")
SRC = r"""
#include "once_per_device.h"
#include <cassert>
#include <cstdio>
int main() {
    rms::OncePerDevice once;
    int calls[3] = {0, 0, 0};
    for (int round = 0; round < 3; ++round)
        for (int d = 0; d < 3; ++d) assert(once(d, [&] { ++calls[d]; return 0; }) == 0);
    assert(calls[0] == 1 && calls[1] == 1 && calls[2] == 1);
    rms::OncePerDevice again;   // a step that failed is tried again, on its own device only
    int n = 0;
    assert(again(0, [&] { ++n; return 0; }) == 0);
    assert(again(1, [&] { ++n; return 7; }) == 7);
    assert(again(1, [&] { ++n; return 0; }) == 0);
    assert(again(1, [&] { ++n; return 7; }) == 0 && n == 3);
    std::puts("ok");
}
"""


def test_once_on_each_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"


def test_function_attributes_are_set_per_device():
    """No device-wide attribute is set under a process-wide flag."""
    src = open(os.path.join(CSRC, "rms_contract.cu")).read()
    at = [m.start() for m in re.finditer("cudaFuncSetAttribute", src)]
    assert at
    for k in at:
        head = src[max(0, k - 900):k]
        assert "opt_in(dev" in head and "call_once" not in head
