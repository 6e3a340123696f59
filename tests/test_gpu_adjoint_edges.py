"""Adjoint gathers and scatters at the edges of the grid: grids of a few cells
(every cell wraps), tiles with a ragged last column of blocks, markers whose
stencils reach ghost columns, ghost rows and the wall row of V.  The mixed
gradient against the FP64 one, the FP64 gradient and its state part against
central differences of the drag along a random direction."""
from __future__ import annotations

import numpy as np
import pytest

from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import CylSpec, GridSpec, Solver, State

pytestmark = pytest.mark.gpu
WALLS, PERIODIC = abi.F8_BC_WALLS, abi.F8_BC_PERIODIC


def _case(shape, bc, where):
    w = configs.c4_adjoint()
    h = 2 * np.pi / shape[1]
    g = GridSpec(3, *shape, shape[0] * h, shape[1] * h, shape[2] * h, bc, 0.1 if bc == WALLS else 0.0)
    r = 1.1 * h
    spot = {"centre": (g.lx / 2, g.ly / 2), "x": (r + 0.6 * h, g.ly / 2), "y": (g.lx / 2, r + 0.75 * h),
            "top": (g.lx / 2, g.ly - r - 1.2 * h)}[where]
    cyls = (CylSpec(*spot, r),)
    st = configs.initial_state(configs.replace(w, grid=g, cyls=cyls))
    rng = np.random.default_rng(5)
    for f in ("u", "v", "w"):
        st.arrays[f] = st.arrays[f] + 0.05 * rng.standard_normal(st.arrays[f].shape)
    # a smooth positive definite C without equal face candidates
    z, y, x = np.meshgrid(*(2 * np.pi * np.arange(-0.5, n + 1) / n for n in shape[::-1]), indexing="ij")
    for m in range(6):
        st.arrays["c"][..., m] = (1.3 if m in (0, 3, 5) else 0.0) + 0.15 * (
            np.sin(x + 0.7 * m) * np.cos(y + 0.3 * m) + np.sin(z + 1.1 * m) * np.cos(x - 0.2 * m))
    return g, w.phys, cyls, st


@pytest.mark.parametrize("shape", [(8, 4, 4), (16, 8, 8), (32, 16, 8)])
@pytest.mark.parametrize("bc,where", [(PERIODIC, "centre"), (PERIODIC, "x"), (PERIODIC, "y"), (WALLS, "centre"),
                                      (WALLS, "y"), (WALLS, "top")])
def test_state_gradient_by_differences(gpu, shape, bc, where):
    """Two Newtonian steps, drag objective: <dJ/dU, d> against (J(U + e d) - J(U - e d)) / 2e.  J is a polynomial in U
    whose cubic and higher terms carry dt^3; with e = 1e-6 truncation (e^2) and rounding (1e-16 |J| / e) are below 1e-6
    of the derivative."""
    g, ph, cyls, st = _case(shape, bc, where)
    ph = configs.replace(ph, beta=1.0)
    rng = np.random.default_rng(6)
    d = {}
    for f in ("u", "v", "w"):
        d[f] = np.zeros(g.halo_shape)
        d[f][1:-1, 1:-1, 1:-1] = rng.standard_normal(g.interior_shape)
    e = 1e-6
    with Solver(gpu, g, ph, cyls, precision=abi.F8_FP64) as s:
        def value(sign):
            t = State(dict(st.arrays))
            for f in d:
                t.arrays[f] = st.arrays[f] + sign * e * d[f]
            s.load(t)
            return s.grad(2, 0)[1]
        fd = (value(1.0) - value(-1.0)) / (2 * e)
        s.load(st)
        ds = s.grad(2, 0, want_dstate=True)[3]
    ad = sum(float(np.sum(ds[f] * d[f])) for f in d)
    assert abs(ad - fd) <= 1e-6 * max(abs(fd), float(np.abs(ds["u"]).max()))


@pytest.mark.parametrize("shape", [(64, 32, 32), (32, 32, 64)])
@pytest.mark.parametrize("bc,where", [(PERIODIC, "x"), (PERIODIC, "centre"), (WALLS, "y"), (WALLS, "top")])
def test_mixed_gradient_against_fp64(gpu, shape, bc, where):
    """Three steps with the polymer, the parameter gradient of both precisions: FP32 adjoint fields, 1e-3 of the largest
    entry (as the other mixed gradient tests)."""
    g, ph, cyls, st = _case(shape, bc, where)
    out = []
    for prec in (abi.F8_FP64, abi.F8_MIXED):
        with Solver(gpu, g, ph, cyls, precision=prec) as s:
            s.load(st)
            out.append(s.grad(3, 2)[2])
    scale = np.abs(out[0]).max()
    assert np.abs(out[0] - out[1]).max() <= 1e-3 * scale
