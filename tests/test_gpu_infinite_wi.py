"""Wi = infinity (no relaxation, no polymer stress) is a valid parameter: the
FP64 step against the oracle, whose divisions by Wi give zero."""
from __future__ import annotations

import numpy as np
import pytest

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_infinite_relaxation_time(gpu, oracle, dim):
    w = configs.replace(configs.c1_2d(), cyls=()) if dim == 2 else configs.replace(configs.c2_3d(), cyls=())
    shape = (16, 8, 1) if dim == 2 else (16, 8, 8)
    g = GridSpec(dim, *shape, *(n * np.pi / 4 for n in shape), abi.F8_BC_PERIODIC, 0.0)
    st = configs.initial_state(configs.replace(w, grid=g, noise=0.2))
    out = []
    for fns in (gpu, oracle):
        with Solver(fns, g, configs.replace(w.phys, wi=float("inf")), (), precision=abi.F8_FP64) as s:
            s.load(st)
            s.step(2, want_drag=False)
            out.append(s.store())
    for f in ("u", "v", "c"):
        assert rel_l2(interior(out[0][f]), interior(out[1][f])) <= 1e-10, f
