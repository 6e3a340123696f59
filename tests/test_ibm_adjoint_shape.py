"""The launch of the IBM transpose (f8_common.cuh), on the CPU: every marker has a
thread, no block more than 128, and no more warps than markers need, so that a
2D box's markers are spread over the chip."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

HARNESS = r"""
#include <cstdio>
#include "f8_common.cuh"
int main() {
    int bad = 0;
    for (int nm : {1, 10, 31, 32, 33, 96, 127, 128, 129, 358, 548, 1368, 5344, 21117, 1000000}) {
        const f8::IbmAdjShape s = f8::ibm_adj_shape(nm);
        const long threads = 32L * s.chunks * s.warps, warps = (nm + 31) / 32;
        bad += threads < nm || s.warps > 4 || s.warps < 1 || s.chunks < 1;
        bad += (long)s.chunks < (warps + 3) / 4;                 // as many blocks as its warps fill
        bad += (long)(s.chunks - 1) * s.warps >= warps;          // no block without markers
    }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_shape(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not Path("/usr/local/cuda/include/cuda_runtime.h").exists():
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "s.cpp", tmp_path / "s"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{ROOT / 'fortran8_gb300' / 'csrc'}", "-I/usr/local/cuda/include",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
