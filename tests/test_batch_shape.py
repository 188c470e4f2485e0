"""The rule that picks a batch's kernel shape, evaluated by the compiler (no GPU):
as many warps as are resident, and the other kernel where none is."""
import os
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent

CASES = """
using namespace apsep;
constexpr int R = 152 * kSegWarps;
static_assert(batch_warps(1, 152, 6 * R) == R);
static_assert(batch_warps(1, 152, 6 * R - 1) == 0, "too few tiles a warp");
static_assert(batch_warps(0, 152, 1 << 22) == 0, "no CTA fits an SM");
static_assert(batch_warps(1, 20, 6 * 400) == 400, "a device of 20 SMs");
static_assert(batch_warps(2, 152, 6 * kMaxRanges) == kMaxRanges, "never more ranges than have words");
static_assert(batch_warps(2, 152, 6 * kMaxRanges - 1) == 0);
int main() {}
"""


def test_batch_warps(tmp_path):
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if cxx is None or not os.path.exists(nvcc):
        pytest.skip("no host compiler or CUDA headers")
    include = pathlib.Path(nvcc).resolve().parent.parent / "include"
    src = tmp_path / "shape.cpp"
    src.write_text('#include "apsep_internal.h"\n' + CASES)
    r = subprocess.run([cxx, "-std=c++17", "-fsyntax-only", "-I", str(include), "-I", str(ROOT / "include"),
                        "-I", str(ROOT / "apsep_gb300" / "csrc"), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
