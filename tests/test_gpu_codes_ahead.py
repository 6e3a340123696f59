"""The FP64 3D step chooses the next step's face candidates beside its solves,
inside one call: several steps of one call against the same steps one call at a
time, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import CylSpec, GridSpec, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 4, 4), (32, 16, 16), (64, 32, 64)])
@pytest.mark.parametrize("bc,ncyl", [(abi.F8_BC_PERIODIC, 0), (abi.F8_BC_PERIODIC, 1), (abi.F8_BC_WALLS, 1)])
def test_steps_of_one_call(gpu, shape, bc, ncyl):
    w = configs.c3_channel()
    h = 2 * np.pi / shape[1]
    g = GridSpec(3, *shape, shape[0] * h, shape[1] * h, shape[2] * h, bc, 0.1 if bc == abi.F8_BC_WALLS else 0.0)
    cyls = (CylSpec(g.lx / 2, g.ly / 2, 0.9 * h),) if ncyl else ()
    st = configs.initial_state(configs.replace(w, grid=g, cyls=cyls))
    st.arrays["u"] = st.arrays["u"] + 0.2 * np.random.default_rng(1).standard_normal(st.arrays["u"].shape)
    out = []
    for calls in ((5,), (1, 1, 1, 1, 1), (2, 3)):
        with Solver(gpu, g, w.phys, cyls, precision=abi.F8_FP64) as s:
            s.load(st)
            drag = [s.step(n)[1] for n in calls]
            out.append((s.store(), None if drag[0] is None else np.concatenate(drag)))
    for other, d in out[1:]:
        for f in ("u", "v", "w", "p", "c", "ax0", "tx0"):
            assert np.array_equal(out[0][0][f], other[f]), f
        assert d is None or np.array_equal(out[0][1], d)
