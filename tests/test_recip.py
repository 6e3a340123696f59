"""The division by a known divisor of the FP64 kernels (f8_recip.cuh) against
the division itself, bit for bit, on the CPU: grid spacings and their squares,
powers of two, random divisors; random, zero, infinite and NaN dividends.  A
random quotient differs from the division with a probability of about 2^-50.
Quotients below 2^-969, where x l itself rounds on the subnormal grid, may be one
unit of the last place off."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

HARNESS = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "f8_recip.cuh"

static bool same(double a, double b) {
    if (a != a || b != b) return a != a && b != b;
    if (b != 0.0 && std::fabs(b) < 0x1p-969 && (a == std::nextafter(b, 0.0) || a == std::nextafter(b, 2 * b))) return true;
    return std::memcmp(&a, &b, 8) == 0;
}

int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> m(1.0, 2.0);
    std::uniform_int_distribution<int> ed(-300, 300), ex(-600, 600);
    const double inf = INFINITY, pi2 = 6.283185307179586;
    std::vector<double> ds{1.0, -1.0, 2.0, 0.5, 3.0, 1.0e-3, 2.0e-5, 1.0 / 3.0, inf, -inf, 0.0, -0.0, (double)NAN, 0x1p-500,
                           std::nextafter(1.0, 2.0), std::nextafter(1.0, 0.0)};
    for (int n = 4; n <= 1024; n *= 2)
        for (double l : {1.0, pi2, 2 * pi2, 0.7})
            for (double f : {1.0, 2.0, 4.0}) { ds.push_back(f * (l / n)); ds.push_back((l / n) * (l / n)); }
    for (int q = 0; q < 4000; ++q) ds.push_back(std::ldexp(m(g), ed(g)) * (q & 1 ? -1 : 1));
    long bad = 0, n = 0, special = 0;
    for (double d : ds) {
        const f8::Recip r = f8::recip(d);
        for (double x : {0.0, -0.0, inf, -inf, (double)NAN, 1.0, -1.0, d, -d, 1.0e300, 1.0e-300}) {
            if (!same(f8::div_by(x, r), x / d)) { ++special; std::printf("special %a / %a: %a, not %a\n", x, d, f8::div_by(x, r), x / d); }
            ++n;
        }
        for (int q = 0; q < 1500; ++q) {
            const double x = std::ldexp(m(g), ex(g)) * (q & 1 ? -1 : 1);
            if (!same(f8::div_by(x, r), x / d)) { if (bad++ < 5) std::printf("%a / %a\n", x, d); }
            ++n;
        }
    }
    std::printf("%ld %ld of %ld\n", bad, special, n);
    return bad || special;
}
"""


def test_quotients(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not Path("/usr/local/cuda/include/cuda_runtime.h").exists():
        pytest.skip("no C++ compiler or CUDA headers")
    src, exe = tmp_path / "recip.cpp", tmp_path / "recip"
    src.write_text(HARNESS)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", f"-I{ROOT / 'fortran8_gb300' / 'csrc'}",
                    "-I/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
