"""The error norm of a trial step (csrc/ionic_common.cuh): the largest ratio of
error and tolerance, whatever the order of the states and however they are dealt
to the four warps that share a cell."""
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "cardiacfoam_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <cmath>
#define __forceinline__ inline
#include "ionic_common.cuh"
int main()
{
    // a line: number of states, then (state, warp, error, tolerance) in the order
    // in which a warp takes its states
    int n;
    while (std::scanf("%d", &n) == 1) {
        cfg::ErrorNorm part[4];
        for (int k = 0; k < n; ++k) {
            int i, w;
            double e, t;
            if (std::scanf("%d %d %la %la", &i, &w, &e, &t) != 4) return 1;
            part[w].take(e, t, i);
        }
        double v = part[0].value();
        for (int w = 1; w < 4; ++w)
            if (part[w].value() > v) v = part[w].value();
        std::printf("%d %la\n", part[0].state, v);
    }
}
"""


def _cases(rng):
    """States whose ratios lie within some ulps of one another, exact ties, zeros,
    and what a diverged trial leaves."""
    for _ in range(300):
        n = int(rng.integers(2, 12))
        tol = np.exp(rng.uniform(-30, 30, n))
        e = tol * np.float64(rng.uniform(0.1, 3.0))
        for i in range(n):
            for _ in range(int(rng.integers(0, 3))):
                e[i] = np.nextafter(e[i], rng.choice([0.0, np.inf]))
        yield e, tol
    yield np.array([0.0, 0.0, 0.0]), np.array([1.0, 2.0, 3.0])
    yield np.array([0.5, 1.0, 2.0, 1.0]), np.array([1.0, 2.0, 4.0, 2.0])
    yield np.array([1.0, np.inf, 3.0, np.inf]), np.array([1.0, 2.0, 3.0, 4.0])
    yield np.array([1.0, np.nan, 3.0]), np.array([1.0, 2.0, np.nan])
    yield np.array([1.0, np.inf, 1e300]), np.array([1.0, np.inf, 1e299])


def _expected(e, tol):
    best, state = None, -1
    for i, (a, t) in enumerate(zip(e, tol)):
        if np.isnan(a) or np.isnan(t) or np.isinf(t) or a == 0:
            continue
        r = np.inf if np.isinf(a) else Fraction(float(a)) / Fraction(float(t))
        if best is None or r > best:
            best, state = r, i
    return state, 0.0 if best is None else float(best)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_norm_does_not_depend_on_the_split(tmp_path):
    """A Fraction's float() is the ratio rounded once, as one division is."""
    src, exe = tmp_path / "n.cpp", tmp_path / "n"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    rng = np.random.default_rng(7)
    lines, want = [], []
    for e, tol in _cases(rng):
        for split in (np.zeros(len(e), int), rng.integers(0, 4, len(e)), np.arange(len(e)) % 4):
            lines.append(f"{len(e)} " + " ".join(
                f"{i} {split[i]} {float(e[i]).hex()} {float(tol[i]).hex()}"
                for i in range(len(e))))
            want.append(_expected(e, tol))
    out = subprocess.run([str(exe)], input="\n".join(lines), text=True, check=True,
                         capture_output=True).stdout.splitlines()
    assert len(out) == len(want)
    for k, (line, got, w) in enumerate(zip(lines, out, want)):
        state, value = got.split()
        assert float.fromhex(value) == w[1], line
        assert k % 3 or int(state) == w[0], line      # one warp: the first such state
