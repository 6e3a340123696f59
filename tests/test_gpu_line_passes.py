"""f8_fft_solve over the lengths and line counts between which the transforms
choose their form (stages in shared memory, passes in registers): every length
of the register passes, both sides of the line count, ragged last blocks."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from .conftest import rel_l2
from fortran8_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 1024, 16), (64, 512, 32), (128, 256, 32), (256, 32, 128), (512, 128, 16),
                                   (1024, 64, 16), (2, 32, 1024), (16, 128, 512), (512, 512, 1), (256, 256, 1), (1024, 1024, 1)])
@pytest.mark.parametrize("lhs", [(0.0, -1.0), (1.0, 1e-4)])
def test_periodic_solve(gpu, shape, lhs):
    nx, ny, nz = shape
    rng = np.random.default_rng(2)
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
    assert rel_l2(phi.cpu().numpy(), np.fft.ifftn(spec).real) <= 1e-12
