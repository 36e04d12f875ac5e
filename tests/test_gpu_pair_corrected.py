"""Float-pair PCG where the explicit correction of the Laplacian is kept in FP64
(FP64 contexts on meshes with their full geometry), against the FP64 PCG of the
same context: rows over the full width of 6, of 4 and over their own length, and
tetrahedra."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib, lv
from cardiacfoam_gb300.mesh import box_mesh, with_box_geometry

# rotated fibres: the correction does not vanish on a box mesh
SIGMA = (0.08, 0.03, 0.01, 0.06, 0.02, 0.05)
H = 5e-4


def _pair_of_runs(make, steps, dt):
    runs = []
    for arithmetic in (lib.PCG_FP64, lib.PCG_FLOAT_PAIRS):
        m = make()
        m.set_pcg_arithmetic(arithmetic)
        iters = []
        for _ in range(steps):
            m.step(dt)
            iters.append(np.asarray(m.stats()[2]).astype(int))
        runs.append((m.vm(), iters))
        m.close()
    return runs


def _compare(runs, bound):
    (va, ia), (vb, ib) = runs
    assert np.ptp(va) > 1e-3                 # the stimulus has left a front
    assert np.max(np.abs(va - vb)) <= bound * np.max(np.abs(va))
    for x, y in zip(ia, ib):
        assert abs(int(x.sum()) - int(y.sum())) <= 2


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(9, 8, 7), (23, 11, 1), (31, 1, 1)], ids=["w6", "w4", "w2"])
def test_corrected_box(gpu_lib, dims):
    """Both solved to 1e-10 in the normalised residual: Vm agrees to what that
    leaves (1e-8 of its largest value, as on plain meshes)."""
    l = [d * H for d in dims]
    mesh = with_box_geometry(box_mesh(*dims, *l), *l)
    box = [((0.0, 0.0, 0.0), (1.5e-3, 1.5e-3, 1.5e-3), 0.0, 2e-3, 5e4)]
    _compare(_pair_of_runs(lambda: api.Monodomain(
        mesh, "TNNP", "epicardialCells", SIGMA, dt=1e-5, boxes=box, stencil=False,
        pcg_tol=1e-10, precision=lib.PRECISION_FP64), 20, 1e-5), 1e-8)


@pytest.mark.gpu
def test_corrected_tetrahedra(gpu_lib):
    """The ventricle of the mixed form's test, in FP64 and within its bound."""
    L = lv.left_ventricle(4, 8, 12, sigma_l=10 * lv.SIGMA_L, sigma_t=10 * lv.SIGMA_T)
    lo, hi = L.apex_box(8e-3)
    _compare(_pair_of_runs(lambda: api.Monodomain(
        L.mesh, "TNNP", "epicardialCells", dt=5e-5, precision=lib.PRECISION_FP64,
        boxes=[(lo, hi, 0.0, 2e-3, 5e4)], tissue_per_cell=L.tissue,
        conductivity_per_cell=L.conductivity, stencil=False), 40, 5e-5), 1e-9)
