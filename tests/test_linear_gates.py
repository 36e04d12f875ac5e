"""Linear gates of the tissue step: the closed form of a Fehlberg step
(csrc/linear_gates.cuh) against the stages themselves, the emitter's list of
linear states, and the FP64 kernels that fold a tissue's constants against the
ones that evaluate them per cell."""
import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cardiacfoam_gb300 import api, lib
from cardiacfoam_gb300.cellml2cuda import cexpr
from cardiacfoam_gb300.cellml2cuda.gates import slope

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "cardiacfoam_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cmath>
#define __forceinline__ inline
#define __fmaf_rn fmaf
#define __fma_rn fma
#include "linear_gates.cuh"
using namespace cfg;
template <int S> static double q(double z) { return lingate::stage_poly<S, double>(z); }
int main()
{
    double z;
    while (std::scanf("%lf", &z) == 1)
        std::printf("%.17g %.17g %.17g %.17g %.17g %.17g %.17g\n", q<1>(z), q<2>(z), q<3>(z),
                    q<4>(z), q<5>(z), lingate::increment_poly<double>(z),
                    lingate::error_poly<double>(z));
}
"""


def fehlberg(z):
    """Stage inputs, increment and embedded error of y' = -b y + a over one
    step with z = -h b, per unit of h k1, summed as the tableau writes them."""
    a = [[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
         [439 / 216, -8.0, 3680 / 513, -845 / 4104],
         [-8 / 27, 2.0, -3544 / 2565, 1859 / 4104, -11 / 40]]
    b = [16 / 135, 0.0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]
    b4 = [25 / 216, 0.0, 1408 / 2565, 2197 / 4104, -1 / 5, 0.0]
    k, q = [1.0], []
    for row in a[1:]:
        q.append(sum(c * x for c, x in zip(row, k)))
        k.append(1.0 + z * q[-1])
    return (q + [sum(c * x for c, x in zip(b, k))] +
            [sum((d - c) * x for c, d, x in zip(b, b4, k))])


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_polynomials_are_the_fehlberg_stages(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    zs = [0.0, -1e-8, -1e-3, -0.1, -0.5, -1.0, -3.0, -20.0, 0.7]
    out = subprocess.run([str(exe)], input="\n".join(map(repr, zs)), text=True, check=True,
                         capture_output=True).stdout
    for z, line in zip(zs, out.splitlines()):
        got, want = [float(v) for v in line.split()], fehlberg(z)
        # the tableau's sums hold terms of size up to 8 |k|, k up to 1 + |z|^5
        scale = 8.0 * (1.0 + abs(z)) ** 5
        assert np.allclose(got, want, rtol=1e-13, atol=16 * 2.0 ** -52 * scale), z


def test_slope_of_gate_expressions():
    for text in ("(CONSTANTS[a] - STATES[y]) / CONSTANTS[t]",
                 "CONSTANTS[a] * (1.0 - STATES[y]) - CONSTANTS[b] * STATES[y]"):
        e = cexpr.parse_expr(text)
        s = slope(e, "y")
        env = {"a": 3.0, "b": 0.5, "t": 4.0}

        def ev(n, y):
            if isinstance(n, cexpr.Num):
                return n.value
            if isinstance(n, cexpr.Ref):
                return y if n.array == "STATES" else env[n.name]
            if isinstance(n, cexpr.Unary):
                return -ev(n.e, y)
            l, r = ev(n.l, y), ev(n.r, y)
            return {"+": l + r, "-": l - r, "*": l * r, "/": l / r if r else 0.0}[n.op]
        assert abs(ev(s, 0.3) - (ev(e, 1.0) - ev(e, 0.0))) < 1e-14, text
    for text in ("STATES[y] * STATES[y]", "CONSTANTS[a] / STATES[y]", "exp(STATES[y])"):
        with pytest.raises(ValueError):
            slope(cexpr.parse_expr(text), "y")


def test_lin_mask_names_the_states_with_a_decay():
    """The bits of LIN_MASK are the states gate_decay() sets, and rhs_tissue()
    assigns the rate of each exactly once, outside any conditional, reading no
    state but that one."""
    n = 0
    for path in sorted((CSRC / "models").glob("*_plain.cuh")):
        text = path.read_text()
        common = (path.parent / path.name.replace("_plain", "")).read_text()
        states = re.search(r"enum State \{ (.*?) \};", common).group(1).split(", ")
        mask = int(re.search(r"LIN_MASK = 0x([0-9a-f]+)ull", text).group(1), 16)
        body = text[text.index("void gate_decay("):]
        gates = re.findall(r"b\[(S_\w+)\] =", body[:body.index("\n}\n")])
        assert [s for i, s in enumerate(states) if mask >> i & 1] == gates, path.name
        assert not mask & 1
        if not mask:
            continue
        rhs = text[text.index("double rhs_tissue("):]
        rhs = rhs[:rhs.index("\n}\n")]
        for g in gates:
            lines = [x for x in rhs.splitlines() if f"dydt[{g}] =" in x]
            assert len(lines) == 1 and lines[0].startswith("    dydt["), (path.name, g)
            reads = set(re.findall(r"\by_(\w+)", lines[0])) - {states[0][2:]}
            assert reads == {g[2:]}, (path.name, g)
            n += 1
    assert n > 50


@pytest.mark.gpu
@pytest.mark.parametrize("solve_vm", [False, True], ids=["tissue", "single cell"])
@pytest.mark.parametrize("n", [1, 31, 33, 129])
@pytest.mark.parametrize("model,tissue", [("TNNP", "mCells"), ("ORd", "myocyte"),
                                          ("ToRORd_dynCl", "endocardialCells")])
def test_folded_constants_equal_per_cell_constants(gpu_lib, model, tissue, n, solve_vm):
    """FP64: scales of one take the kernel with per-cell constants, no scales
    the kernel of the tissue; same equations, so equal to round-off (the bound
    is the one the oracle comparisons use for adaptive steps)."""
    dt, steps = 2e-5, 3
    im = []
    for scales in (None, np.ones((6, n))):
        g = api.IonicModel(model, tissue, n, dt, solve_vm_within_ode=solve_vm,
                           ode=api.ode_desc(max_steps=10 ** 6), scales=scales)
        out = np.zeros(n)
        vm = np.linspace(-0.086, 0.03, n)
        for s in range(steps):
            g.solveODE(s * dt, dt, None if solve_vm else vm, out)
        im.append((out.copy(), g.states()))
        g.close()
    (a, ya), (b, yb) = im
    assert np.all(np.isfinite(a))
    assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a))
    assert np.max(np.abs(ya - yb) / np.maximum(np.abs(yb), 1e-12)) <= 1e-9
