"""The cable solve of a Purkinje network at the edges of its launch: a chain (one
node a level), a star (a level wider than the block), a level of one warp and one
more, and a network that shared memory does not hold."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api

H = 2.5e-4


def _edges(shape):
    rng = np.random.default_rng(2)
    if shape == "pair":
        pairs = [(0, 1)]
    elif shape == "chain":
        pairs = [(k, k + 1) for k in range(300)]
    elif shape.startswith("star"):
        n = int(shape[4:])
        pairs = [(0, k) for k in range(1, n + 1)]
    else:                                    # random tree, nodes in random order
        n = int(shape[4:])
        label = np.concatenate([[0], 1 + rng.permutation(n - 1)])
        pairs = [(int(label[rng.integers(max(0, k - 60), k)]), int(label[k])) for k in range(1, n)]
    return [(a, b, H * rng.uniform(0.8, 1.2), rng.uniform(0.5, 1.5)) for a, b in pairs]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", ["pair", "chain", "star32", "star33", "star1500", "tree900",
                                   "tree9000"])
def test_cable_shapes(gpu_lib, oracle, shape):
    """Vm of every node after some steps under a root stimulus, within 1e-11 of
    the field's scale: the tree's matrix is diagonally dominant, so roundings
    of 1e-16 do not grow over its levels."""
    e = _edges(shape)
    dt = 1e-5
    g = api.Purkinje(e, "BuenoOrovio", "epicardialCells", dt=dt, root_stimulus=(0, 0.0, 2e-3, 5e5))
    o = oracle.Purkinje(e, "BuenoOrovio", 1, dt, root_stimulus=(0.0, 2e-3, 5e5))
    for step in (dt, dt, 0.5 * dt, dt):
        g.step(step)
        o.advance(step)
    vg, vo = g.vm(), o.vm()
    assert np.max(np.abs(vo - vo[-1])) > 0
    assert np.max(np.abs(vg - vo)) <= 1e-11 * np.max(np.abs(vo))
    g.close()
