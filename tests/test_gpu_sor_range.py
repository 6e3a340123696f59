"""The stopping test of the mixed step's SOR solve over the exponent range of
FP32: right-hand sides whose squares FP32 cannot hold (residuals of 1e-23 and
less, of 1e20 and more).  The sweeps are linear, so the mixed solve takes as many
as the FP64 solve of the same fields (within one, as at unit scale), and both
give the same velocities to the solve's tolerance: a residual of 1e-5 of the
right-hand side in the longest wave moves the velocity by 1e-5 times the ratio
of the largest wavenumber to the least, 35 on 64 cells."""
from __future__ import annotations

import numpy as np
import pytest

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 8, 8), (64, 64, 32), (64, 64, 64)])      # one block, a cluster, the whole chip
@pytest.mark.parametrize("scale", [2.0 ** -90, 2.0 ** -60, 1.0, 2.0 ** 30])
def test_scaled_flow(gpu, shape, scale):
    w = configs.c2_3d()
    h = 2 * np.pi / shape[1]
    g = GridSpec(3, *shape, shape[0] * h, shape[1] * h, shape[2] * h, abi.F8_BC_PERIODIC, 0.0)
    st = configs.initial_state(configs.replace(w, grid=g, flow="uniform", noise=1e-2))
    rng = np.random.default_rng(3)
    for f in ("u", "v", "w"):
        st.arrays[f] = scale * rng.standard_normal(st.arrays[f].shape)
    # a step short enough that convection stays small beside the velocity
    ph = configs.replace(w.phys, beta=1.0, sor_itrmax=2000, dt=w.phys.dt * min(1.0, 0.01 / scale))
    out = {}
    for prec in (abi.F8_FP64, abi.F8_MIXED):
        with Solver(gpu, g, ph, (), precision=prec, poisson=abi.F8_POISSON_SOR) as s:
            s.load(st)
            status, _ = s.step(1, want_drag=False)
            assert status == abi.F8_OK
            out[prec] = (s.store(), s.diagnostics().poisson_iters)
    assert out[abi.F8_FP64][1] > 5
    assert abs(out[abi.F8_MIXED][1] - out[abi.F8_FP64][1]) <= 1
    for f in ("u", "v", "w"):
        assert rel_l2(interior(out[abi.F8_MIXED][0][f]), interior(out[abi.F8_FP64][0][f])) <= 4e-4, f
