"""One cell, the smallest system of the persistent solve.  Its normFactor is of
rounding size, so iteration counts say nothing there; Vm does."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.mesh import box_mesh

SIGMA = (0.1334, 0.0, 0.0, 0.0176, 0.0, 0.0176)
H = 5e-4
BOX = [((0.0, 0.0, 0.0), (1.5e-3, 1.5e-3, 1.5e-3), 0.0, 2e-3, 5e4)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [lib.PRECISION_FP64, lib.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
@pytest.mark.parametrize("stencil", [True, False], ids=["stencil", "ell"])
def test_one_cell_in_pairs(gpu_lib, stencil, precision):
    """Float pairs against FP64, the persistent solve against the kernel
    sequence: Vm within 1e-8, the bound of the larger systems."""
    mesh = box_mesh(1, 1, 1, H, H, H)
    vm = []
    for arithmetic, persistent in ((lib.PCG_FLOAT_PAIRS, True), (lib.PCG_FP64, True),
                                   (lib.PCG_FP64, False)):
        m = api.Monodomain(mesh, "TNNP", "epicardialCells", SIGMA, dt=1e-5, boxes=BOX,
                           stencil=stencil, pcg_tol=1e-10, precision=precision)
        m.set_pcg_arithmetic(arithmetic)
        m.set_persistent(persistent)
        for _ in range(8):
            m.step(1e-5)
        vm.append(m.vm())
        m.close()
    assert np.all(np.isfinite(vm)) and vm[0][0] > -0.083       # the stimulus has risen
    assert np.max(np.abs(vm[0] - vm[2])) <= 1e-8 * np.max(np.abs(vm[2]))
    assert np.max(np.abs(vm[1] - vm[2])) <= 1e-8 * np.max(np.abs(vm[2]))
