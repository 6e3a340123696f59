"""The comparison of the grid barrier's arrival counters (f8_common.cuh), on the
CPU: a block waits until the counter has reached its own count, across the
wrap of both at 2^32 (about 14 million sweeps on 152 SMs; sor_itrmax has no upper limit)."""
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
    for (unsigned blocks : {1u, 2u, 152u, 1024u})
        for (unsigned start : {0u, 1000000u, 0x7fffff00u, 0x80000000u, 0xfffffff0u, 0xffffffffu})
            for (unsigned round = 1; round <= 4; ++round) {
                const unsigned target = start + round * blocks;
                for (unsigned back = 1; back <= blocks; ++back) bad += !f8::behind(target - back, target);   // not all here
                for (unsigned on = 0; on <= blocks; ++on) bad += f8::behind(target + on, target);            // all, some already at the next
            }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_arrivals(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not Path("/usr/local/cuda/include/cuda_runtime.h").exists():
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "b.cpp", tmp_path / "b"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{ROOT / 'fortran8_gb300' / 'csrc'}", "-I/usr/local/cuda/include",
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
