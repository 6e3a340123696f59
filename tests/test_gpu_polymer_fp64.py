"""The FP64 polymer update against the oracle where its branches differ: the
diagonal pivots of the usual Newton system, the exchanged rows of a strongly
sheared one, and the edges of its 32 x 4 blocks."""
from __future__ import annotations

import numpy as np
import pytest

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed", [1.0, 300.0])   # dt |grad u|: 1e-2 and a few units
@pytest.mark.parametrize("name,shape", [("c2_3d", (4, 4, 4)), ("c2_3d", (64, 8, 8)), ("c3_channel", (32, 8, 4)),
                                        ("c1_2d", (16, 16, 1)), ("c1_2d", (64, 4, 1))])
def test_update_matches_oracle(gpu, oracle, name, shape, speed):
    w = configs.scaled(getattr(configs, name)(), *shape)
    st = configs.initial_state(w)
    rng = np.random.default_rng(4)
    for f in ("u", "v", "w") if w.grid.dim == 3 else ("u", "v"):
        st[f][:] = speed * rng.standard_normal(st[f].shape)
    n = w.grid.dim
    a = rng.standard_normal(st["c"].shape[:3] + (n, n))
    c = a @ np.swapaxes(a, -1, -2) + np.eye(n)
    st["c"][:] = np.stack([c[..., p, q] for p in range(n) for q in range(p, n)], -1)
    res = []
    for fns in (gpu, oracle):
        with Solver(fns, w.grid, w.phys, (), precision=abi.F8_FP64) as s:
            s.load(st)
            s.step(1, want_drag=False)
            res.append((s.store()["c"], s.diagnostics().newton_iters))
    assert rel_l2(interior(res[0][0]), interior(res[1][0])) <= 1e-10
    assert res[0][1] == res[1][1]
