"""The IBM transpose with more markers than one block takes (128): the last block
and its last warp part full, two cylinders whose markers share warps.  FP64
gradients of the drag after two Newtonian steps against central differences: of
the state along a random direction (within 1e-6, as the other test of it) and of
the cylinder centres (within 1e-4, as the other tests of them)."""
from __future__ import annotations

import numpy as np
import pytest

from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import CylSpec, GridSpec, Solver, State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,shape,radii,least", [(2, (32, 32, 1), (1.2,), 129), (2, (64, 64, 1), (1.3, 0.9), 641),
                                                   (2, (128, 64, 1), (1.1, 1.1), 641), (3, (64, 32, 4), (1.3, 0.9), 193),
                                                   (3, (32, 32, 8), (1.25,), 129)])
@pytest.mark.parametrize("bc", [abi.F8_BC_PERIODIC, abi.F8_BC_WALLS])
def test_many_markers(gpu, dim, shape, radii, least, bc):
    w = configs.c1_2d() if dim == 2 else configs.c4_adjoint()
    h = 2 * np.pi / shape[1]
    g = GridSpec(dim, *shape, shape[0] * h, shape[1] * h, shape[2] * h, bc, 0.0)
    spots = [(g.lx / 2 + 0.0123, g.ly / 2 + 0.0371)] if len(radii) == 1 else [(g.lx * 0.27 + 0.0123, g.ly * 0.3 + 0.0371),
                                                                              (g.lx * 0.7 + 0.0211, g.ly * 0.68 + 0.0173)]
    cyls = tuple(CylSpec(x, y, r) for (x, y), r in zip(spots, radii))
    st = configs.initial_state(configs.replace(w, grid=g, cyls=cyls))
    rng = np.random.default_rng(8)
    vel = ("u", "v", "w")[:dim]
    for f in vel:
        st.arrays[f] = st.arrays[f] + 0.05 * rng.standard_normal(st.arrays[f].shape)
    ph = configs.replace(w.phys, beta=1.0)
    d = {}
    for f in vel:
        d[f] = np.zeros(g.halo_shape)
        d[f][1:-1, 1:-1, 1:-1] = rng.standard_normal(g.interior_shape)
    e = 1e-6

    def value(cy, s0):
        with Solver(gpu, g, ph, cy, precision=abi.F8_FP64) as s:
            s.load(s0)
            return s.grad(2, 0)[1]

    with Solver(gpu, g, ph, cyls, precision=abi.F8_FP64) as s:
        assert len(s.markers()) >= least
        s.load(st)
        _, _, dp, ds, _ = s.grad(2, 0, want_dstate=True)
    along = []
    for sign in (1.0, -1.0):
        t = State(dict(st.arrays))
        for f in vel:
            t.arrays[f] = st.arrays[f] + sign * e * d[f]
        along.append(value(cyls, t))
    fd = (along[0] - along[1]) / (2 * e)
    ad = sum(float(np.sum(ds[f] * d[f])) for f in vel)
    assert abs(ad - fd) <= 1e-6 * max(abs(fd), float(np.abs(ds["u"]).max()))
    centre = []
    for l in range(len(cyls)):
        for key in ("xc", "yc"):
            v = []
            for sign in (1.0, -1.0):
                moved = [configs.replace(c, **({key: getattr(c, key) + sign * e} if q == l else {})) for q, c in enumerate(cyls)]
                v.append(value(tuple(moved), st))
            centre.append((v[0] - v[1]) / (2 * e))
    assert np.abs(dp[3:] - centre).max() <= 1e-4 * np.abs(centre).max()
