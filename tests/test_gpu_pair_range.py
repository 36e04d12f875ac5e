"""The bidomain's float-pair solve where (z, r) falls below the range whose
reciprocals floats hold."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.mesh import box_mesh, with_box_geometry

SIGMA_I = (0.1334, 0.0, 0.0, 0.0176, 0.0, 0.0176)
SIGMA_E = (0.62, 0.0, 0.0, 0.24, 0.0, 0.24)


@pytest.mark.gpu
def test_nearly_uniform_potential(gpu_lib):
    """A resting cube of 20^3 cells (Aliev-Panfilov: no current at rest) under a
    source that moves 27 cells by 1e-10 V.  In the scaled phiE system (z, r)
    starts at 8e-22 and ends, at 1e-8 in the normalised residual, near 3e-40
    (both from a FP64 solve of the same system); 1 / x overflows below 2.9e-39.
    Vm is solved to 1e-3, which bounds what phiE differs by."""
    n, h, dt = 20, 5e-4, 2e-5
    mesh = with_box_geometry(box_mesh(n, n, n, n * h, n * h, n * h), n * h, n * h, n * h)
    box = [((0.0, 0.0, 0.0), (3.01 * h, 3.01 * h, 3.01 * h), 0.0, 1.0, 1e-10 * 1400 / dt)]
    runs = []
    for arithmetic in (lib.PCG_FP64, lib.PCG_FLOAT_PAIRS):
        bd = api.Bidomain(mesh, "AlievPanfilov", "myocyte", sigma_i=SIGMA_I, sigma_e=SIGMA_E,
                          dt=dt, vm0=-0.08, pcg_tol=1e-3, phie_tol=1e-8, boxes=box,
                          ref_point=(0.0, 0.0, 0.0))
        bd.set_pcg_arithmetic(arithmetic)
        for _ in range(2):                           # phiE follows Vm a step behind
            bd.step(dt)                              # raises where a solve fails
        runs.append((bd.vm(), bd.phie()))
        bd.close()
    (v0, p0), (v1, p1) = runs
    assert np.all(np.isfinite(v1)) and np.all(np.isfinite(p1))
    assert 1e-11 < np.ptp(v0) < 1e-9
    assert 1e-13 < np.max(np.abs(p0)) < 1e-10
    assert np.max(np.abs(p1 - p0)) <= 1e-2 * np.max(np.abs(p0))
