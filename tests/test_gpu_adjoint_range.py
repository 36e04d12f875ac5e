"""The mixed adjoint's reverse on adjoints far from one: a misfit against targets
that large (the gradients are proportional to them), against the FP64 form."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.mesh import box_mesh

H = 2.5e-4


@pytest.mark.gpu
@pytest.mark.parametrize("size", [1.0, 1e29, 1e33])
def test_reverse_range(gpu_lib, size):
    """What differs is the FP32 right-hand side: the bound is that of the small
    sheets (1e-4 of the largest value) where the misfit does not depend on the
    trace's own rounding, which at targets of this size it does not."""
    nx = 65
    mesh = box_mesh(nx, 1, 1, nx * H, H, H)
    probes = np.arange(0, nx, 9)
    box = [((0.0, 0.0, 0.0), (nx * H, H, H), 0.0, 2e-3, 5e4)]
    rng = np.random.default_rng(6)
    a, b = (0.2 * rng.standard_normal(nx) for _ in range(2))
    out = []
    for precision in (lib.PRECISION_FP64, lib.PRECISION_MIXED):
        p = api.AdjointProblem(mesh, 6, 1e-5, probes, 3, checkpoint_every=4, substeps=5,
                               boxes=box, precision=precision)
        _, trace = p.forward(a, b, 0.1334, 0.0176)
        # the misfit is size everywhere, whatever the trace
        p.set_target(np.asarray(trace) - size)
        p.forward(a, b, 0.1334, 0.0176)
        out.append([np.asarray(g) for g in p.backward()])
        p.close()
    for x, y in zip(*out):
        assert np.all(np.isfinite(x)) and np.all(np.isfinite(y))
        assert np.max(np.abs(x)) > 0
        assert np.max(np.abs(x - y)) <= 1e-4 * np.max(np.abs(x))
