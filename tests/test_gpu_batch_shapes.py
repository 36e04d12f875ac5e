"""The mixed batch kernel (state and stage data in shared memory) at the edges of
its blocks: one cell, a warp and a block and one cell more; against the FP64
form."""
import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib

TISSUE = {"TNNP": "epicardialCells", "ORd": "myocyte", "ToRORd_dynCl": "endocardialCells"}


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 33, 65])
@pytest.mark.parametrize("model", list(TISSUE))
def test_mixed_batch_shapes(gpu_lib, model, n):
    """Twenty steps from rest: states within 1e-4 of each state's largest value
    (unit roundoff 6e-8 times some hundred operations a right-hand side), and
    every cell of a batch with equal scales alike, bit for bit."""
    dt, steps = 1e-5, 20
    stimuli = [api.stimulus_desc(10.0, 1000.0, 1.0, 0.0, 1)] * n
    out = []
    for precision in (lib.PRECISION_FP64, lib.PRECISION_MIXED):
        b = api.BatchCells(model, TISSUE[model], dt, stimuli, np.full(n, steps * dt),
                           precision=precision, ode=api.ode_desc(max_steps=10 ** 6))
        b.run()
        out.append(np.asarray(b.states()))
        b.close()
    y64, y32 = out
    assert y32.shape == y64.shape and np.all(np.isfinite(y32))
    assert np.all(y32 == y32[:, :1])
    scale = np.max(np.abs(y64), axis=1, keepdims=True)
    assert np.all(np.abs(y32 - y64) <= 1e-4 * scale + 1e-12)
