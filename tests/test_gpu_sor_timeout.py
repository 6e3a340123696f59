"""The bounded waits of the SOR solve's grid barrier.  A small program launches
the kernel with a limit of zero cycles, so that the first block to arrive gives
up (the kernel ends by itself, as each wait is bounded), and reads the time-out
flag; the same buffers then give the solution that a context without a time-out
gives.  And a step whose solve reports a time-out (the flag set on the host, by a
library loaded before the CUDA runtime) returns F8_ERR_CUDA; a load and a step on
the same context then work."""
from __future__ import annotations

import json
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "fortran8_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <vector>
#include "f8_sor.cuh"
using namespace f8;

template <typename T>
int run() {
    Geo g{};
    g.nx = 32; g.ny = 16; g.nz = 16; g.sx = 34; g.sy = 18; g.sz = 18; g.dim = 3;
    g.dx = g.dy = g.dz = 0.25;
    const size_t cs = (size_t)g.sx * g.sy * g.sz, ni = (size_t)g.nx * g.ny * g.nz;
    std::vector<T> q(ni), p0(cs), p1(cs);
    double er = 0;
    for (size_t n = 0; n < ni; ++n) { q[n] = (T)std::sin(0.37 * n + 0.01 * (n % 7)); er += (double)q[n] * q[n]; }
    T *Phi, *R; double *er0; SorSum<T> *part; int *flag, f[4];
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
    if (cudaMalloc(&Phi, cs * sizeof(T)) || cudaMalloc(&R, ni * sizeof(T)) || cudaMalloc(&er0, 8) ||
        cudaMalloc(&part, 2 * SOR_MAX_BLOCKS * sizeof(SorSum<T>)) || cudaMalloc(&flag, 16)) return 2;
    cudaMemcpy(R, q.data(), ni * sizeof(T), cudaMemcpyHostToDevice);
    cudaMemcpy(er0, &er, 8, cudaMemcpyHostToDevice);
    SorArgs<T> a{};
    a.Phi = Phi; a.R = R; a.er0 = er0; a.part = part; a.flag = flag;
    a.om = (T)1.8; a.bx = a.by = a.bz = 16; a.b0 = 96;
    a.rb0 = recip(96.0);
    a.eps = 1e-4; a.itrmax = 300;
    int status[3], late[3], iters[3];
    for (int n = 0; n < 3; ++n) {
        a.wait = n == 1 ? 0 : SOR_WAIT_CYCLES;
        cudaMemset(Phi, 0, cs * sizeof(T));
        status[n] = sor_sweeps(a, g, sms, 1, 0);
        if (!status[n]) status[n] = cudaDeviceSynchronize();
        cudaMemcpy(f, flag, 16, cudaMemcpyDeviceToHost);
        late[n] = f[2]; iters[n] = f[1];
        if (n != 1) cudaMemcpy((n ? p1 : p0).data(), Phi, cs * sizeof(T), cudaMemcpyDeviceToHost);
    }
    const bool ok = !status[0] && !status[1] && !status[2] && !late[0] && late[1] == 1 && !late[2] && iters[0] > 1 &&
                    iters[0] == iters[2] && p0 == p1;
    std::printf("status %d %d %d late %d %d %d sweeps %d %d\n", status[0], status[1], status[2], late[0], late[1], late[2],
                iters[0], iters[2]);
    return ok ? 0 : 1;
}

int main() { return run<double>() | run<float>(); }
"""

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static void *fn(const char *name) {
    static void *h;
    if (!h) h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    return h ? dlsym(h, name) : 0;
}
static int armed, *flags, seen;
int cudaMemcpyAsync(void *dst, const void *src, size_t n, int kind, void *s) {
    int (*f)(void *, const void *, size_t, int, void *) = (int (*)(void *, const void *, size_t, int, void *))fn("cudaMemcpyAsync");
    if (armed && n == 12 && kind == 2) flags = (int *)dst;      /* converged, iteration, time-out */
    return f(dst, src, n, kind, s);
}
int cudaStreamSynchronize(void *s) {
    int (*f)(void *) = (int (*)(void *))fn("cudaStreamSynchronize"), e = f(s);
    if (flags) { flags[2] = 1; flags = 0; ++seen; }
    return e;
}
void shim_arm(int on) { armed = on; }
int shim_seen(void) { return seen; }
"""

CHILD = r"""
import ctypes, json, sys
import numpy as np
from fortran8_gb300 import abi, configs, lib
from fortran8_gb300.solver import F8Error, GridSpec, Solver

shim = ctypes.CDLL(sys.argv[1])
w = configs.c2_3d()
g = GridSpec(3, 32, 16, 16, 8.0, 4.0, 4.0, 0, 0.0)
st = configs.initial_state(configs.replace(w, grid=g, cyls=(), noise=0.1))
out = []
for prec in (0, 1):
    with Solver(lib.functions(), g, w.phys, (), precision=prec, poisson=abi.F8_POISSON_SOR) as s:
        s.load(st)
        s.step(2, want_drag=False)
        ref = s.store()
        s.load(st)
        shim.shim_arm(1)
        try:
            s.step(2, want_drag=False)
            status = 0
        except F8Error as e:
            status = e.status
        shim.shim_arm(0)
        s.load(st)
        s.step(2, want_drag=False)
        got = s.store()
        out.append([status, shim.shim_seen(), all(np.array_equal(got[f], ref[f]) for f in ("u", "v", "w", "p", "c"))])
print(json.dumps(out))
"""


def test_wait_runs_out(gpu, tmp_path):
    from fortran8_gb300 import build
    src, exe = tmp_path / "late.cu", tmp_path / "late"
    src.write_text(PROGRAM)
    subprocess.run([build._nvcc(), *build.ARCH, "-O2", "-std=c++17", "-diag-suppress", "177", f"-I{CSRC}", str(src),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_step_reports_it(gpu, tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    assert cc, "no C compiler"
    so = tmp_path / "shim.so"
    (tmp_path / "shim.c").write_text(SHIM)
    (tmp_path / "child.py").write_text(CHILD)
    subprocess.run([cc, "-shared", "-fPIC", "-O1", str(tmp_path / "shim.c"), "-o", str(so), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, str(tmp_path / "child.py"), str(so)], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    rec = json.loads(r.stdout.splitlines()[-1])
    assert [x[0] for x in rec] == [4, 4] and [x[1] for x in rec] == [1, 2] and all(x[2] for x in rec), rec
