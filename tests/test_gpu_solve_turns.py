"""f8_fft_solve from several threads: calls on one device take turns at its
workspace, a call on another device does not wait for them.  One GPU serves: a
library loaded before the CUDA runtime holds a thread that asks for it at the end
of its first stream synchronisation (its kernels have ended by then), and tells
another thread that its device is number 1."""
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
#include <unistd.h>
static void *fn(const char *name) {
    static void *h;
    if (!h) h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
    return h ? dlsym(h, name) : 0;
}
static volatile int held, released;
static __thread int hold, device = -1;
int cudaStreamSynchronize(void *s) {
    int (*f)(void *) = (int (*)(void *))fn("cudaStreamSynchronize"), e = f(s);
    if (hold) {
        hold = 0;
        held = 1;
        for (int n = 0; n < 5000 && !released; ++n) usleep(1000);     /* 5 s at most */
        held = 0;
    }
    return e;
}
int cudaGetDevice(int *d) {
    int (*f)(int *) = (int (*)(int *))fn("cudaGetDevice"), e = f(d);
    if (!e && device >= 0) *d = device;
    return e;
}
void shim_hold(void) { hold = 1; released = 0; }
void shim_device(int d) { device = d; }
int shim_held(void) { return held; }
void shim_release(void) { released = 1; }
"""

CHILD = r"""
import ctypes, json, sys, threading, time
import numpy as np
import torch
from fortran8_gb300 import lib

shim = ctypes.CDLL(sys.argv[1])
solve = lib.functions()["fft_solve"]
n = (32, 16, 8)
q = [torch.randn(n[::-1], dtype=torch.float64, device="cuda") for _ in range(3)]
p = [torch.zeros_like(x) for x in q]
ptr = [(a.data_ptr(), b.data_ptr()) for a, b in zip(q, p)]
call = lambda k: solve(*n, 2.0, 1.0, 0.5, *ptr[k], 1.0, 1e-4)
assert call(0) == 0
ref = []
for k in range(3):
    assert call(k) == 0
    ref.append(p[k].clone())
    p[k].zero_()
torch.cuda.synchronize()
ended = {}

def first():
    shim.shim_hold()
    ended["st0"] = call(0)
    ended["first"] = time.monotonic()

def other(name, k, device):
    shim.shim_device(device)
    ended["st%d" % k] = call(k)
    ended[name] = time.monotonic()

a = threading.Thread(target=first)
a.start()
while not shim.shim_held():
    time.sleep(0.001)
same = threading.Thread(target=other, args=("same", 1, -1))
far = threading.Thread(target=other, args=("far", 2, 1))
same.start()
far.start()
far.join(3.0)
res = {"far_while_held": "far" in ended and bool(shim.shim_held()), "same_while_held": "same" in ended}
shim.shim_release()
for t in (a, same, far):
    t.join()
res["same_after"] = ended["same"] >= ended["first"] - 0.05
res["status"] = [ended["st%d" % k] for k in range(3)]
res["equal"] = [bool(torch.equal(p[k], ref[k])) for k in range(3)]
print(json.dumps(res))
"""


def test_turns(gpu, tmp_path):
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
    res = json.loads(r.stdout.splitlines()[-1])
    assert res["far_while_held"] and not res["same_while_held"], res
    assert res["status"] == [0, 0, 0] and all(res["equal"]) and res["same_after"], res
