"""The mixed spectral solves over every line length and plane split they are
built for: NX 32 to 512, wall planes of NZ 32 to 256 in one CTA and over a
cluster, planes smaller than the scan's buffer, ragged last row blocks."""
from __future__ import annotations

import numpy as np
import pytest

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu

WALLS, PERIODIC = abi.F8_BC_WALLS, abi.F8_BC_PERIODIC


@pytest.mark.parametrize("shape,bc,uwall", [
    ((32, 4, 32), WALLS, 0.0), ((64, 16, 32), WALLS, 0.3), ((128, 8, 64), WALLS, 0.0), ((256, 32, 128), WALLS, 0.0),
    ((512, 8, 256), WALLS, 0.2), ((32, 256, 64), WALLS, 0.0), ((32, 256, 128), WALLS, 0.0), ((32, 256, 256), WALLS, 0.1),
    ((512, 4, 8), PERIODIC, 0.0), ((256, 32, 4), PERIODIC, 0.0), ((128, 4, 16), PERIODIC, 0.0), ((32, 64, 8), PERIODIC, 0.0)])
def test_mixed_solves_in_a_step(gpu, shape, bc, uwall):
    """Two Newtonian steps, the mixed velocity against FP64: the increments of
    the step are FP32, 1e-5 of the velocity bounds their rounding."""
    w = configs.c3_channel()
    h = 2 * np.pi / shape[1]
    g = GridSpec(3, *shape, shape[0] * h, shape[1] * h, shape[2] * h, bc, uwall)
    ph = configs.replace(w.phys, beta=1.0, dt=1e-4)
    st = configs.initial_state(configs.replace(w, grid=g))
    out = []
    for prec in (abi.F8_FP64, abi.F8_MIXED):
        with Solver(gpu, g, ph, (), precision=prec) as s:
            s.load(st)
            s.step(2, want_drag=False)
            out.append(s.store())
    for f in ("u", "v", "w"):
        assert rel_l2(interior(out[1][f]), interior(out[0][f])) <= 1e-5, f
