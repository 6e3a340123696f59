"""Device memory of an FP64 wall context: the state, its work arrays, one spectrum
per velocity component (the wall solves work in place), the Thomas tables of the
three systems and the queue of the eigen tests, to within the allocator's
granularity (2 MB for each of some 60 arrays; a spectrum has 68 MB)."""
from __future__ import annotations

import numpy as np
import pytest

from fortran8_gb300 import abi, configs
from fortran8_gb300.solver import GridSpec, Solver

pytestmark = pytest.mark.gpu


def test_wall_context(gpu):
    import torch
    nx, ny, nz = 512, 128, 128
    w = configs.c3_channel()
    h = 2 * np.pi / ny
    g = GridSpec(3, nx, ny, nz, nx * h, ny * h, nz * h, abi.F8_BC_WALLS, 0.0)
    with Solver(gpu, g, w.phys, (), precision=abi.F8_FP64):
        pass                                     # the library's own arrays are in place
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with Solver(gpu, g, w.phys, (), precision=abi.F8_FP64):
        used = free - torch.cuda.mem_get_info()[0]
    halo, cells, modes = (nx + 2) * (ny + 2) * (nz + 2), nx * ny * nz, (nx // 2 + 1) * nz * (ny + 2)
    # U V W P Phi U* V* W*, C transposed, f Ua Va Wa, C twice; histories, forces, viscous terms, right-hand sides
    fields = 8 * ((8 + 6 + 4 + 12) * halo + 15 * cells)
    need = fields + 3 * 16 * modes + 3 * 3 * 8 * modes + 12 * nx * (ny + 2) * nz + cells
    assert used <= need + 120 * 2**20, (used / cells, need / cells)
