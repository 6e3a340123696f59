"""The double-float filter of the FP64 eigen test (f8_codes_filter.cuh).

CPU: the kernel's own routines, compiled for the host with the CUDA intrinsics
replaced by their IEEE operations, decide a direction only where the FP64
evaluation of Vieta's formula (fenep.f90:169-242, 425-444) decides the same,
over generic, strongly stretched, nearly isotropic, nearly repeated, indefinite,
equal and out-of-range tensors.  GPU: the codes of one step equal the oracle's
on random SPD fields at the edges of the kernel's tiles (32 x 8 cells); the
y direction of a wall's first row is left out, whose ghost is the linear
extrapolation, so that its three candidates are equal up to rounding.
"""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import Solver

CSRC = Path(__file__).resolve().parents[1] / "fortran8_gb300" / "csrc"

SHIM = r"""
#pragma once
#include <algorithm>
#include <cmath>
#define __device__
#define __host__
#define __forceinline__ inline
struct float2 { float x, y; };
inline float2 make_float2(float a, float b) { return {a, b}; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float2 __fadd2_rn(float2 a, float2 b) { return {a.x + b.x, a.y + b.y}; }
inline float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y)}; }
inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
"""

HARNESS = r"""
#include "f8_codes_filter.cuh"
using namespace f8;
extern "C" void choose(long n, const double *c0, const double *cm, const double *cp, int *out) {
    for (long q = 0; q < n; ++q) {
        codes::CellC c;
        for (int m = 0; m < 6; ++m) c.c[m] = df_from_d(c0[6 * q + m]);
        codes::cell_split(c);
        df2 dv[6];
        for (int m = 0; m < 6; ++m) {
            const df a = df_from_d(cm[6 * q + m]), b = df_from_d(cp[6 * q + m]);
            dv[m] = df2_sub(df2{make_float2(c.c[m].hi, b.hi), make_float2(c.c[m].lo, b.lo)},
                            df2{make_float2(a.hi, c.c[m].hi), make_float2(a.lo, c.c[m].lo)});
        }
        out[q] = codes::choose(c, dv);
    }
}
"""


def vieta(a):
    a0, a1, a2, a3, a4, a5 = a
    A2 = -(a0 + a3 + a5)
    A1 = a0 * a3 + a3 * a5 + a5 * a0 - a4 * a4 - a2 * a2 - a1 * a1
    A0 = -(a0 * a3 * a5 + a1 * a4 * a2 + a1 * a4 * a2 - a0 * a4 * a4 - a1 * a1 * a5 - a2 * a3 * a2)
    p = A1 - (A2 * A2) / 3.0
    q = A0 - A1 * A2 / 3.0 + 2.0 * (A2 * A2 * A2) / 27.0
    t = (q / 2) * (q / 2) + (p / 3) * (p / 3) * (p / 3)
    v = 2.0 * np.sqrt(-p / 3.0) * np.cos(np.arccos(3.0 * q / (2.0 * p) * np.sqrt(-3.0 / p)) / 3.0 + 2 * np.pi / 3) - A2 / 3.0
    return np.where(t >= 0.0, -100.0, v)


def fp64_codes(cm, c0, cp):
    faces = ((c0 * 3 / 2 - cp / 2, c0 / 2 + cp / 2), (cm / 2 + c0 / 2, -cm / 2 + c0 * 3 / 2),
             (cm / 4 + c0 - cp / 4, -cm / 4 + c0 + cp / 4))
    m = [np.fmin(vieta(p.T), vieta(n.T)) for p, n in faces] + [np.zeros(len(c0))]
    m = np.stack(m)
    return np.argmax(np.where(np.isnan(m), -np.inf, m), axis=0)


def six(a):
    return np.stack([a[:, 0, 0], a[:, 0, 1], a[:, 0, 2], a[:, 1, 1], a[:, 1, 2], a[:, 2, 2]], -1)


def tensors(kind, rng, n):
    q = np.linalg.qr(rng.standard_normal((n, 3, 3)))[0]
    if kind == "stretched":
        ev = np.stack([np.full(n, 0.7), 0.7 + rng.random(n), 10 ** rng.uniform(0, 3, n)], -1)
    elif kind == "isotropic":
        ev = 1 + 10 ** rng.uniform(-8, -1, (n, 1)) * rng.standard_normal((n, 3))
    elif kind == "repeated":
        ev = np.stack([np.full(n, 0.7), 0.7 + 10 ** rng.uniform(-9, -1, n), 10 ** rng.uniform(-1, 2, n)], -1)
    elif kind == "indefinite":
        ev = rng.standard_normal((n, 3))
    else:
        ev = rng.uniform(0.3, 5, (n, 3))
    return q @ (ev[:, :, None] * np.eye(3)) @ np.swapaxes(q, 1, 2), np.ptp(ev, axis=1)


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    d = tmp_path_factory.mktemp("filter")
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", f"-I{d}", f"-I{CSRC}", "-shared", "-fPIC",
                    str(d / "h.cpp"), "-o", str(d / "h.so")], check=True)
    fn = C.CDLL(str(d / "h.so")).choose

    def run(cm, c0, cp):
        a = [np.ascontiguousarray(x) for x in (c0, cm, cp)]
        out = np.zeros(len(c0), np.int32)
        fn(C.c_long(len(c0)), *[x.ctypes.data_as(C.c_void_p) for x in a], out.ctypes.data_as(C.c_void_p))
        return out
    return run


@pytest.mark.parametrize("kind", ["generic", "stretched", "isotropic", "repeated", "indefinite"])
@pytest.mark.parametrize("slope", ["random", "nearly linear", "equal", "zero neighbour"])
def test_filter_decides_as_fp64(choose, kind, slope):
    rng = np.random.default_rng(7)
    n = 30000
    c0, spread = tensors(kind, rng, n)
    amp = (10 ** rng.uniform(-6, -0.3, n) * spread)[:, None, None]
    d = [amp * (e + np.swapaxes(e, 1, 2)) / 2 for e in rng.standard_normal((2, n, 3, 3))]
    if slope == "nearly linear":
        d[1] = d[0] * (1 + 10 ** rng.uniform(-9, -1, (n, 1, 1)))
    if slope == "equal":
        d = [0 * d[0], 0 * d[1]]
    c0, cm, cp = six(c0), six(c0 - d[0]), six(c0 + d[1])
    if slope == "zero neighbour":
        cm = 0 * cm
    with np.errstate(all="ignore"):
        want = fp64_codes(cm, c0, cp)
    got = choose(cm, c0, cp)
    assert np.array_equal(got[got >= 0], want[got >= 0])


def test_filter_leaves_extremes_to_fp64(choose):
    rng = np.random.default_rng(8)
    c0, _ = tensors("generic", rng, 64)
    c0 = six(c0)
    for scale in (0.0, 1e-30, 1e-8, 1e13, 1e300, np.inf, np.nan):
        with np.errstate(all="ignore"):
            s = c0 * scale
        assert np.all(choose(s, s, s) == -1)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,walls", [((4, 4, 4), False), ((32, 8, 4), False), ((64, 16, 8), True), ((8, 4, 16), True)])
def test_codes_equal_the_oracle(gpu, oracle, shape, walls):
    w = configs.scaled(configs.c3_channel() if walls else configs.c2_3d(), *shape)
    st = configs.initial_state(w)
    rng = np.random.default_rng(9)
    c, _ = tensors("stretched", rng, st["c"][..., 0].size)
    st["c"][:] = six(c).reshape(st["c"].shape)
    out = []
    for fns in (gpu, oracle):
        with Solver(fns, w.grid, w.phys, (), precision=abi.F8_FP64) as s:
            s.load(st)
            s.step(1, want_drag=False)
            out.append(s.selection_codes())
            if walls:
                out[-1][:, [1, -2]] &= 0b110011
    assert np.array_equal(*out)
