"""The persistent PCG kernels at the edges of their launch shapes: one cell, a
partly filled warp and block, exactly one row per thread of every SM's block,
and one row more (the next block size, then rows in turn), in FP64 and in float
pairs; against the kernel sequence (monodomain), FP64 against float pairs
(bidomain) and central differences (adjoint)."""
import numpy as np
import pytest
import torch

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.mesh import box_mesh, with_box_geometry

SIGMA = (0.1334, 0.0, 0.0, 0.0176, 0.0, 0.0176)
SIGMA_E = (0.62, 0.0, 0.0, 0.24, 0.0, 0.24)
H = 5e-4
# rows per SM: one block of 128, 256, 384, 448 and 512 threads, two of 512
EDGES = ["1", "31", "129", "128/sm", "128/sm+1", "256/sm+1", "384/sm", "384/sm+1", "448/sm+1",
         "512/sm+1", "1024/sm+1"]


def _mesh(edge, geometry=True):
    """A sheet of at least the wanted rows (exactly them where a row of 152
    divides them, else a ragged one)."""
    per, _, more = edge.partition("/sm")
    n = int(per)
    if "/sm" in edge:
        n *= torch.cuda.get_device_properties(0).multi_processor_count
    if more:
        ny = int(np.sqrt(n)) | 1
        nx = n // ny + 1                     # nx ny > n
    else:
        nx, ny = (n, 1) if n < 1000 else (n // 64, 64)
    mesh = box_mesh(nx, ny, 1, nx * H, ny * H, H)
    return with_box_geometry(mesh, nx * H, ny * H, H) if geometry else mesh, nx, ny


BOX = [((0.0, 0.0, 0.0), (1.5e-3, 1.5e-3, 1.5e-3), 0.0, 2e-3, 5e4)]


def _shapes():
    # One cell has a normFactor of rounding size, which the pairs' residual never
    # falls below: Vm agrees, the iteration counts do not.
    one = pytest.mark.xfail(strict=True, reason="normFactor of a single cell is rounding")
    return [pytest.param(e, p, marks=[one] if e == "1" and p else [],
                         id=f"{'pairs' if p else 'fp64'}-{e}")
            for p in (False, True) for e in EDGES]


@pytest.mark.gpu
@pytest.mark.parametrize("edge,pairs", _shapes())
@pytest.mark.parametrize("stencil", [True, False], ids=["stencil", "ell"])
def test_monodomain_shapes(gpu_lib, edge, pairs, stencil):
    """The persistent solve against the kernel sequence: the same solve up to
    the order of sums (and the pairs' 48 bits), so Vm agrees to what the
    solver tolerance of 1e-10 leaves."""
    mesh, _, _ = _mesh(edge, geometry=False)
    runs = []
    for persistent in (True, False):
        m = api.Monodomain(mesh, "TNNP", "epicardialCells", SIGMA, dt=1e-5, boxes=BOX,
                           stencil=stencil, pcg_tol=1e-10)
        m.set_pcg_arithmetic(lib.PCG_FLOAT_PAIRS if pairs and persistent else lib.PCG_FP64)
        m.set_persistent(persistent)
        iters = []
        for _ in range(8):
            m.step(1e-5)
            iters.append(np.asarray(m.stats()[2]).astype(int))
        runs.append((m.vm(), iters))
        m.close()
    (v0, i0), (v1, i1) = runs
    assert np.max(np.abs(v0 - v1)) <= 1e-8 * np.max(np.abs(v1))
    for a, b in zip(i0, i1):
        assert abs(int(a.sum()) - int(b.sum())) <= 2


@pytest.mark.gpu
@pytest.mark.parametrize("edge", EDGES[1:-1])
@pytest.mark.parametrize("stencil", [4, 6], ids=["2d", "3d"])
def test_bidomain_shapes(gpu_lib, edge, stencil):
    """Float pairs against FP64 from the same start, both systems to 1e-9 in
    the normalised residual: they differ by that times the condition number,
    which for the largest sheet (280 cells across) is 4 280^2 / pi^2 = 3e4."""
    mesh, nx, ny = _mesh(edge)
    if stencil == 6:
        nz = 3
        nx = nx // nz + 1
        mesh = with_box_geometry(box_mesh(nx, ny, nz, nx * H, ny * H, nz * H),
                                 nx * H, ny * H, nz * H)
    runs = []
    for arithmetic in (lib.PCG_FP64, lib.PCG_FLOAT_PAIRS):
        bd = api.Bidomain(mesh, "TNNP", "epicardialCells", sigma_i=SIGMA, sigma_e=SIGMA_E,
                          dt=2e-5, pcg_tol=1e-9, phie_tol=1e-9, phie_max_iter=4000, n_outer=1,
                          ref_point=(0.0, 0.0, 0.0), boxes=BOX)
        bd.set_pcg_arithmetic(arithmetic)
        for _ in range(3):
            bd.step(2e-5)
        runs.append((bd.vm(), bd.phie()))
        bd.close()
    for a, b in zip(*runs):
        assert np.max(np.abs(a - b)) <= 4e-5 * np.max(np.abs(b))


@pytest.mark.gpu
@pytest.mark.parametrize("edge", ["129", "128/sm", "128/sm+1", "256/sm+1"])
def test_adjoint_shapes(gpu_lib, edge):
    """One directional derivative against central differences (1e-5 as in the
    small sheet's test)."""
    mesh, nx, ny = _mesh(edge, geometry=False)
    n = nx * ny
    rng = np.random.default_rng(4)
    probes = rng.choice(n, 8, replace=False)
    p = api.AdjointProblem(mesh, 24, 1e-5, probes, 8, checkpoint_every=6, substeps=5,
                           boxes=[((0.0, 0.0, 0.0), (nx * H, ny * H, H), 0.0, 2e-3, 5e4)])
    a, b = (0.1 * rng.standard_normal(n) for _ in range(2))
    _, target = p.forward(0 * a, 0 * b, 0.15, 0.03)
    p.set_target(target)
    J, _ = p.forward(a, b, 0.1334, 0.0176)
    ga, gb, gs = p.backward()
    assert J > 0 and np.all(np.isfinite(ga)) and np.all(np.isfinite(gb))
    va, vb, eps = np.sign(ga), np.sign(gb), 1e-6
    ad = ga @ va + gb @ vb + gs @ np.array([0.1, 0.1])
    jp, jm = (p.forward(a + e * va, b + e * vb, 0.1334 + 0.1 * e, 0.0176 + 0.1 * e)[0]
              for e in (eps, -eps))
    fd = (jp - jm) / (2 * eps)
    assert abs(fd - ad) <= 1e-5 * abs(fd) + 1e-14, (fd, ad)
