"""Mixed batches of the size production populations have (beyond a warp per SM,
at what one SM holds with all states in shared memory, and one cell more): a
cell's result does not depend on how many others run with it, bit for bit, agrees
with the FP64 form, and a failing solve is reported with its cell."""
import re

import numpy as np
import pytest
import torch

from cardiacfoam_gb300 import api, lib

TISSUE = {"TNNP": "epicardialCells", "ORd": "myocyte", "ToRORd_dynCl": "endocardialCells"}
DT, STEPS = 1e-5, 20
ODE = dict(max_steps=10 ** 6)


def _population(n):
    rng = np.random.default_rng(11)
    scales = np.exp(rng.uniform(np.log(0.5), np.log(2.0), (6, n)))
    end = DT * rng.integers(STEPS // 2, STEPS + 1, n)
    end[::97] = 0.0
    end[-1] = STEPS * DT
    return scales, end


def _run(model, scales, end, precision=lib.PRECISION_MIXED, chunk=0, ode=ODE):
    stimuli = [api.stimulus_desc(10.0, 1000.0, 1.0, 0.0, 1)] * len(end)
    b = api.BatchCells(model, TISSUE[model], DT, stimuli, end, precision=precision,
                       scales=scales, ode=api.ode_desc(**ode), chunk=chunk)
    try:
        b.run()
        return np.asarray(b.states()), b.results(), b.stats()[1]
    finally:
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("per_sm,more", [(32, 1), (192, 0), (192, 1)])
@pytest.mark.parametrize("model", list(TISSUE))
def test_population_size(gpu_lib, model, per_sm, more):
    """FP32 against FP64 from rest as in the small batches (1e-4 of each state's
    largest value)."""
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    scales, end = _population(n)
    y, res, steps = _run(model, scales, end)
    assert np.all(np.isfinite(y)) and steps == int(np.round(end / DT).sum())
    some = np.unique(np.r_[0:33, n // 2:n // 2 + 33, n - 33:n])
    part = scales[:, some], end[some]
    y1, res1, _ = _run(model, *part)
    assert np.array_equal(y[:, some], y1)
    for a, b in zip(res, res1):
        assert np.array_equal(a[some], b, equal_nan=True)
    yc, _, _ = _run(model, scales, end, chunk=7)
    assert np.array_equal(y, yc)
    last, _, _ = _run(model, scales[:, -1:], end[-1:])
    assert np.array_equal(y[:, -1:], last)
    y64, _, _ = _run(model, *part, precision=lib.PRECISION_FP64)
    scale = np.max(np.abs(y64), axis=1, keepdims=True)
    assert np.all(np.abs(y1 - y64) <= 1e-4 * scale + 1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("model", list(TISSUE))
def test_failure_in_a_population(gpu_lib, model):
    n = 192 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    scales, end = _population(n)
    with pytest.raises(lib.CfgError) as e:
        _run(model, scales, end, ode=dict(max_steps=1, abs_tol=1e-12, rel_tol=1e-12))
    assert e.value.code == lib.CFG_ERR_ODE_STEPS
    m = re.search(r"cell (\d+)", str(e.value))
    assert m and 0 <= int(m.group(1)) < n
