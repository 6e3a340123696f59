"""f8_load / f8_store of a mixed context without a step: U and V come back as the
sum of the two floats nearest to them, C as floats, over the whole range of
exponents, ties and zeros."""
from __future__ import annotations

import numpy as np
import pytest

from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu


def _values(shape, rng):
    x = rng.standard_normal(shape) * 10.0 ** rng.integers(-44, 37, shape)
    b = x.view(np.uint64)
    tie = rng.integers(0, 4, shape)
    b = np.where(tie == 1, (b & ~np.uint64(0x1fffffff)) | np.uint64(0x10000000), b)      # half way between floats
    b = np.where(tie == 2, b & ~np.uint64(0x1fffffff), b)                                # floats
    x = b.view(np.float64).copy()
    x.flat[::7], x.flat[3::11] = 0.0, -0.0
    return x


@pytest.mark.parametrize("dim,shape", [(3, (8, 4, 4)), (3, (32, 16, 8)), (2, (16, 8, 1))])
def test_round_trip(gpu, dim, shape):
    rng = np.random.default_rng(3)
    w = configs.c2_3d() if dim == 3 else configs.c1_2d()
    h = 2 * np.pi / shape[1]
    g = GridSpec(dim, *shape, shape[0] * h, shape[1] * h, shape[2] * h if dim == 3 else h, abi.F8_BC_PERIODIC, 0.0)
    st = configs.initial_state(configs.replace(w, grid=g, cyls=()))
    for f in ("u", "v", "c"):
        st.arrays[f] = _values(st.arrays[f].shape, rng)
    with Solver(gpu, g, w.phys, (), precision=abi.F8_MIXED) as s:
        s.load(st)
        out = s.store()
    inner = (slice(1, -1),) * 3
    with np.errstate(over="ignore", under="ignore"):
        for f in ("u", "v"):
            x = st.arrays[f][inner]
            hi = x.astype(np.float32)
            lo = (x - hi.astype(np.float64)).astype(np.float32)
            assert np.array_equal(out[f][inner], hi.astype(np.float64) + lo.astype(np.float64)), f
        assert np.array_equal(out["c"][inner], st.arrays["c"][inner].astype(np.float32).astype(np.float64))
