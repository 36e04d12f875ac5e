"""The shape that the autotuner reports is the one it keeps."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.mesh import box_mesh

SIGMA = (0.1334, 0.0, 0.0, 0.0176, 0.0, 0.0176)


@pytest.mark.gpu
def test_rule_that_shares_cells_is_reported_as_such(gpu_lib):
    """FP64, a few tiles of 32 cells: four warps a tile take about half of the
    time of one warp a tile, which is what every explicit block gives."""
    dt = 1e-5
    m = api.Monodomain(box_mesh(8, 8, 3, 0.004, 0.004, 0.0015), "TNNP", "epicardialCells", SIGMA,
                       dt=dt, precision=lib.PRECISION_FP64)
    m.run(dt, 4)
    block, cpt, ms = m.autotune()
    assert (block, cpt) == (0, 1) and ms > 0
    m.close()
    n = 192
    out = []
    for shape in (None, (block, cpt)):
        ion = api.IonicModel("TNNP", "epicardialCells", n, dt, precision=lib.PRECISION_FP64)
        if shape:
            ion.set_launch(*shape)               # a reported shape is accepted
        vm, im = np.linspace(-0.085, 0.02, n), np.zeros(n)
        for k in range(3):
            ion.solveODE(k * dt, dt, vm, im)
        out.append(im)
        ion.close()
    assert np.array_equal(*out)
