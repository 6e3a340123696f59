"""Tolerances that are zero, negative or NaN: no step passes the reference's tests
(sqrt(..) < eps, fenep.f90:575, 885-896), so every cell takes newton_itrmax
iterations and the SOR solve sor_itrmax sweeps; and one whose square underflows.
One FP64 step against the oracle: Newton counts exactly (its operations are the
oracle's), fields to the rounding of the summation orders."""
from __future__ import annotations

import numpy as np
import pytest

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu
EPS = [0.0, -1e-3, float("nan"), 1e-200]


def _state(w, g):
    st = configs.initial_state(configs.replace(w, grid=g, cyls=()))
    rng = np.random.default_rng(4)
    for f in ("u", "v") + (("w",) if g.dim == 3 else ()):
        st.arrays[f] = st.arrays[f] + 0.1 * rng.standard_normal(st.arrays[f].shape)
    return st


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("dim", [2, 3])
def test_newton(gpu, oracle, dim, eps):
    w = configs.c1_2d() if dim == 2 else configs.c2_3d()
    shape = (16, 8, 1) if dim == 2 else (16, 8, 8)
    h = 2 * np.pi / 8
    g = GridSpec(dim, *shape, *(n * h for n in shape), abi.F8_BC_PERIODIC, 0.0)
    ph = configs.replace(w.phys, newton_eps=eps, newton_itrmax=7)
    out = []
    for fns in (gpu, oracle):
        with Solver(fns, g, ph, (), precision=abi.F8_FP64) as s:
            s.load(_state(w, g))
            status, _ = s.step(1, want_drag=False)
            d = s.diagnostics()
            out.append((status, d.newton_iters, d.newton_unconverged, s.store()))
    assert out[0][:3] == out[1][:3]
    assert eps > 0 or out[0][0] == abi.F8_WARN_NEWTON
    for f in ("u", "v", "c"):
        assert rel_l2(interior(out[0][3][f]), interior(out[1][3][f])) <= 1e-10, f


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("prec,shape", [(0, (16, 8, 8)), (1, (16, 8, 8)), (1, (64, 64, 32)), (1, (64, 64, 64))])
def test_sor(gpu, prec, shape, eps):
    w = configs.c2_3d()
    h = 2 * np.pi / shape[1]
    g = GridSpec(3, *shape, *(n * h for n in shape), abi.F8_BC_PERIODIC, 0.0)
    ph = configs.replace(w.phys, beta=1.0, sor_eps=eps, sor_itrmax=400)
    with Solver(gpu, g, ph, (), precision=prec, poisson=abi.F8_POISSON_SOR) as s:
        s.load(_state(w, g))
        status, _ = s.step(1, want_drag=False)
        assert status == abi.F8_WARN_SOR and s.diagnostics().poisson_iters == 401
