"""The line transforms and the tabulated Thomas solves at the edges of their
launch shapes: one column or row pair per block, blocks of a few threads, long
lines, one-point directions, ragged last blocks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from .conftest import interior, rel_l2
from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2, 1), (4, 4, 4), (1024, 4, 2), (4, 1024, 1), (8, 2, 512), (64, 64, 8), (256, 32, 32)])
@pytest.mark.parametrize("lhs", [(0.0, -1.0), (1.0, 1e-4)])
def test_periodic_solve(gpu, shape, lhs):
    nx, ny, nz = shape
    rng = np.random.default_rng(1)
    q = rng.standard_normal((nz, ny, nx))
    box = (2.0, 1.5, 1.0)
    dq = torch.tensor(q, device="cuda")
    phi = torch.empty_like(dq)
    torch.cuda.synchronize()
    assert gpu["fft_solve"](nx, ny, nz, *box, dq.data_ptr(), phi.data_ptr(), *lhs) == abi.F8_OK
    lam = sum(np.reshape(2 * (1 - np.cos(np.arange(n) * (2 * np.pi / n))) / (l / n) ** 2, s)
              for n, l, s in ((nx, box[0], (1, 1, -1)), (ny, box[1], (1, -1, 1)), (nz, box[2], (-1, 1, 1))))
    den = lhs[0] + lhs[1] * lam
    spec = np.fft.fftn(q)
    spec = np.where(np.abs(den) < 1e-16, 0.0, spec / np.where(np.abs(den) < 1e-16, 1.0, den))
    assert rel_l2(phi.cpu().numpy(), np.fft.ifftn(spec).real) <= 1e-13


@pytest.mark.parametrize("dim,shape,uwall", [(3, (4, 4, 4), 0.0), (3, (64, 4, 16), 0.3), (3, (8, 256, 4), 0.0),
                                             (2, (128, 8, 1), 0.5), (2, (4, 512, 1), 0.0)])
def test_wall_solves_in_a_step(gpu, oracle, dim, shape, uwall):
    """Two Newtonian channel steps (no cylinders): FP64 against the oracle, the
    mixed velocity against FP64 (the pressure of this nearly uniform flow is at
    the level of the FP32 increments)."""
    w = configs.c3_channel()
    h = 2 * np.pi / shape[1]
    g = GridSpec(dim, *shape, shape[0] * h, shape[1] * h, shape[2] * h if dim == 3 else h, abi.F8_BC_WALLS, uwall)
    ph = configs.replace(w.phys, beta=1.0, dt=1e-4)
    st = configs.initial_state(configs.replace(w, grid=g))
    out = []
    for fns, prec in ((gpu, abi.F8_FP64), (oracle, abi.F8_FP64), (gpu, abi.F8_MIXED)):
        with Solver(fns, g, ph, (), precision=prec) as s:
            s.load(st)
            s.step(2, want_drag=False)
            out.append(s.store())
    for f in ("u", "v", "p") + (("w",) if dim == 3 else ()):
        a, b, m = (interior(o[f]) for o in out)
        assert rel_l2(a, b) <= 1e-10, f
        assert f == "p" or rel_l2(m, a) <= 1e-5, f
