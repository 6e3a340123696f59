"""The one-kernel SOR solve at the edges of its forms: one block, a cluster that
is not full, the largest cluster grid, the cooperative grid (more cells than
131072), 2D, walls and uneven extents.  FP64 at a tight tolerance against the
spectral solve; mixed against FP64 at the reference's tolerance."""
from __future__ import annotations

import numpy as np
import pytest

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,shape,walls", [(3, (4, 4, 4), False), (3, (16, 8, 32), True), (3, (64, 64, 32), False),
                                             (3, (64, 64, 64), True), (3, (64, 8, 32), True), (2, (64, 32, 1), False),
                                             (2, (32, 16, 1), True)])
def test_sor_solve(gpu, dim, shape, walls):
    w = configs.c3_channel() if walls else configs.c2_3d()
    h = 2 * np.pi / shape[1]
    g = GridSpec(dim, *shape, shape[0] * h, shape[1] * h, shape[2] * h if dim == 3 else h,
                 abi.F8_BC_WALLS if walls else abi.F8_BC_PERIODIC, 0.0)
    st = configs.initial_state(configs.replace(w, grid=g, flow="poiseuille" if walls else "uniform", noise=1e-2))
    out = {}
    for name, prec, pois, eps in (("fft", 0, 0, 1e-5), ("tight", 0, 1, 1e-11), ("sor", 0, 1, 1e-5), ("mixed", 1, 1, 1e-5)):
        if name == "mixed" and dim == 2:
            continue      # the 2D mixed step has the FFT solver only
        ph = configs.replace(w.phys, beta=1.0, sor_eps=eps)
        with Solver(gpu, g, ph, (), precision=prec, poisson=pois) as s:
            s.load(st)
            status, _ = s.step(2, want_drag=False)
            assert status == abi.F8_OK
            out[name] = (s.store(), s.diagnostics().poisson_iters)
    for f in ("u", "v") + (("w",) if dim == 3 else ()):
        a = {k: interior(o[0][f]) for k, o in out.items()}
        assert rel_l2(a["tight"], a["fft"]) <= 1e-8, f
        if dim == 3:
            assert rel_l2(a["mixed"], a["sor"]) <= 1e-5, f
    if dim == 3:
        assert abs(out["mixed"][1] - out["sor"][1]) <= 1
