"""A step that fails between the fork and the join of its side streams.  The
failure is made on the host: a small library loaded before the CUDA runtime
returns an error from the k-th cudaStreamWaitEvent instead of making the call
(every wait of a call of three steps in turn: the FP64 candidates beside the
solves, the mixed branches launched directly and under capture).  The call
returns F8_ERR_CUDA with no kernel left on a side stream, and a load and two
steps on the same context then give what a fresh context gives, bit for bit."""
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

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdint.h>

static void *fn(const char *name) {
    static void *h;
    if (!h) h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    return h ? dlsym(h, name) : 0;
}
static void *streams[64];
static int nstreams, countdown, waits;

int cudaStreamCreateWithFlags(void **s, unsigned flags) {
    int (*f)(void **, unsigned) = (int (*)(void **, unsigned))fn("cudaStreamCreateWithFlags");
    int e = f(s, flags);
    if (!e && nstreams < 64) streams[nstreams++] = *s;
    return e;
}
int cudaStreamCreateWithPriority(void **s, unsigned flags, int priority) {
    int (*f)(void **, unsigned, int) = (int (*)(void **, unsigned, int))fn("cudaStreamCreateWithPriority");
    int e = f(s, flags, priority);
    if (!e && nstreams < 64) streams[nstreams++] = *s;
    return e;
}
int cudaStreamWaitEvent(void *s, void *ev, unsigned flags) {
    int (*f)(void *, void *, unsigned) = (int (*)(void *, void *, unsigned))fn("cudaStreamWaitEvent");
    ++waits;
    if (countdown && --countdown == 0) return 999;
    return f(s, ev, flags);
}
void shim_fail_at(int k) { countdown = k; waits = 0; }
int shim_waits(void) { return waits; }
void shim_forget(void) { nstreams = 0; }
/* streams with work left, but the first one created (the context's own) */
int shim_busy(void) {
    int (*f)(void *) = (int (*)(void *))fn("cudaStreamQuery"), n = 0;
    for (int q = 1; q < nstreams; ++q) n += f(streams[q]) != 0;
    return n;
}
int shim_streams(void) { return nstreams; }
"""

CHILD = r"""
import ctypes, json, sys
import numpy as np
from fortran8_gb300 import abi, configs, lib
from fortran8_gb300.solver import CylSpec, F8Error, GridSpec, Solver

shim = ctypes.CDLL(sys.argv[1])
gpu = lib.functions()
out = []
for name, bc, prec, poisson, shape in (("fp64 box", 0, 0, 0, (64, 64, 64)), ("fp64 channel", 1, 0, 0, (64, 32, 64)),
                                       ("mixed box", 0, 1, 0, (64, 32, 32)), ("mixed channel", 1, 1, 0, (64, 32, 32)),
                                       ("mixed sor", 1, 1, 1, (32, 16, 16))):
    w = configs.c3_channel()
    h = 2 * np.pi / shape[1]
    g = GridSpec(3, *shape, *(n * h for n in shape), bc, 0.0)
    cyls = (CylSpec(g.lx / 2, g.ly / 2, 2.5 * h),)
    st = configs.initial_state(configs.replace(w, grid=g, cyls=cyls))
    fields = ("u", "v", "w", "p", "c", "ax0", "tx0")
    shim.shim_fail_at(0)
    with Solver(gpu, g, w.phys, cyls, precision=prec, poisson=poisson) as s:
        s.load(st)
        d = s.step(2)[1]
        ref = s.store()
        s.load(st)
        s.step(3)
    with Solver(gpu, g, w.phys, cyls, precision=prec, poisson=poisson) as s:
        s.load(st)
        shim.shim_fail_at(0)
        s.step(3)
        n = shim.shim_waits()
    rec = {"name": name, "waits": n, "status": [], "busy": [], "same": []}
    for k in range(1, n + 1):
        shim.shim_forget()
        with Solver(gpu, g, w.phys, cyls, precision=prec, poisson=poisson) as s:
            s.load(st)
            shim.shim_fail_at(k)
            try:
                s.step(3)
                rec["status"].append(0)
            except F8Error as e:
                rec["status"].append(e.status)
            rec["busy"].append(shim.shim_busy())
            shim.shim_fail_at(0)
            s.load(st)
            d2 = s.step(2)[1]
            got = s.store()
            rec["same"].append(all(np.array_equal(got[f], ref[f]) for f in fields) and np.array_equal(d, d2))
    rec["streams"] = shim.shim_streams()
    out.append(rec)
print(json.dumps(out))
"""


def test_failed_waits(gpu, tmp_path):
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
    for rec in json.loads(r.stdout.splitlines()[-1]):
        assert rec["waits"] > 0 and rec["streams"] > 1, rec
        assert all(s == 4 for s in rec["status"]), rec
        assert not any(rec["busy"]), rec
        assert all(rec["same"]), rec
