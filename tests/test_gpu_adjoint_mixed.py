"""The mixed adjoint's ionic kernels (float-pair sums, V-only values apart) against
the FP64 form: sheets around a block of 64 cells and beyond the reverse's
resident threads, the least and most substeps, every tissue."""
import numpy as np
import pytest
import torch

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.mesh import box_mesh

H = 2.5e-4


@pytest.mark.gpu
@pytest.mark.parametrize("nx,substeps,tissue", [
    (3, 1, "epicardialCells"), (64, 5, "mCells"), (65, 16, "endocardialCells"),
    (0, 2, "epicardialCells")], ids=["part-warp", "block", "block+1", "beyond-resident"])
def test_mixed_sums_against_fp64(gpu_lib, nx, substeps, tissue):
    """A few steps, of substeps short enough for the explicit stages (2 us: the
    gate m of a resting cell), from rest under a stimulus of the whole sheet, so that nothing
    is amplified: what differs is the FP32 right-hand side (unit roundoff 6e-8,
    some hundred operations in a row, differences of nearly equal terms in the
    currents), bounded by 1e-4 of the largest value."""
    # a persistent grid has at most 32 blocks of 64 threads per SM
    ny = 1 if nx else 256
    nx = nx or (torch.cuda.get_device_properties(0).multi_processor_count * 2048) // 256 + 1
    n = nx * ny
    mesh = box_mesh(nx, ny, 1, nx * H, ny * H, H)
    probes = np.arange(0, n, max(1, n // 7))
    box = [((0.0, 0.0, 0.0), (nx * H, ny * H, H), 0.0, 2e-3, 5e4)]
    rng = np.random.default_rng(6)
    a, b = (0.2 * rng.standard_normal(n) for _ in range(2))
    out, target = [], None
    for precision in (lib.PRECISION_FP64, lib.PRECISION_MIXED):
        p = api.AdjointProblem(mesh, 6, substeps * 2e-6, probes, 3, checkpoint_every=4, substeps=substeps,
                               tissue=tissue, boxes=box, precision=precision)
        if target is None:
            _, target = p.forward(0 * a, 0 * b, 0.15, 0.03)
            target = 0.97 * np.asarray(target)
        p.set_target(target)
        J, trace = p.forward(a, b, 0.1334, 0.0176)
        out.append((np.asarray(trace), *(np.asarray(g) for g in p.backward())))
        p.close()
    for x, y in zip(*out):
        assert np.max(np.abs(y)) > 0
        assert np.max(np.abs(x - y)) <= 1e-4 * np.max(np.abs(y))
