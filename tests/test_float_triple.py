"""Sums in three floats (csrc/float_pair.cuh, Acc3), compiled for the host: what
the mixed adjoint carries over a step holds more bits than a sum in FP64."""
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "cardiacfoam_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cuda_runtime.h>
#undef __forceinline__
#define __forceinline__ inline
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fdiv_rn(float a, float b) { return a / b; }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
static float __double2float_rn(double a) { return float(a); }
static float __uint2float_rn(unsigned a) { return float(a); }
static long long __double_as_longlong(double a) { long long b; std::memcpy(&b, &a, 8); return b; }
static unsigned __float_as_uint(float a) { unsigned b; std::memcpy(&b, &a, 4); return b; }
static float __uint_as_float(unsigned a) { float b; std::memcpy(&b, &a, 4); return b; }
static float __shfl_down_sync(unsigned, float a, int) { return a; }
#include "float_pair.cuh"
int main()
{
    int n;
    while (std::scanf("%d", &n) == 1) {
        cfg::fp::Acc3 s;
        for (int k = 0; k < n; ++k) {
            float w, x;
            if (std::scanf("%a %a", &w, &x) != 2) return 1;
            if (w == 1.0f) s.add(x);
            else s.add_prod(w, x);
        }
        std::printf("%la\n", s.join());
    }
}
"""


# a step's weights over their common denominator, and floats of all 24 bits
WEIGHTS = np.array([33440, 146432, 142805, -50787, 10260, 0.1, -7 / 3], np.float32).astype(float)


def _cases(rng):
    for _ in range(400):
        n = int(rng.integers(1, 61))
        w = np.where(rng.random(n) < 0.3, 1.0, rng.choice(WEIGHTS, n))
        x = (rng.standard_normal(n) * 10.0 ** rng.uniform(-6, 6, n)).astype(np.float32)
        if rng.random() < 0.3:                       # all but cancelling
            w[n // 2:], x[n // 2:] = -w[:n - n // 2], x[:n - n // 2]
        yield w, x


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_triple_sums(tmp_path):
    """Within the rounding of the result to a double and 2^-57 of the terms'
    magnitudes.  The second float holds the errors of the first, at most 60 2^-24
    of the terms, the third those of the second, at most 2 60 2^-24 of it, and a
    rounding of the third is 2^-24 of that: 2 60 2 60 60 2^-72 < 2^-52 at the
    very worst, random signs leave its root; a sum in FP64 has 60 2^-53."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    inc = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), "-I", str(inc),
                    str(src), "-o", str(exe)], check=True)
    rng = np.random.default_rng(3)
    cases = list(_cases(rng))
    text = "\n".join(f"{len(w)} " + " ".join(f"{float(a).hex()} {float(b).hex()}"
                                             for a, b in zip(w, x)) for w, x in cases)
    out = subprocess.run([str(exe)], input=text, text=True, check=True,
                         capture_output=True).stdout.split()
    assert len(out) == len(cases)
    for (w, x), got in zip(cases, out):
        terms = [Fraction(float(a)) * Fraction(float(b)) for a, b in zip(w, x)]
        total, size = sum(terms), sum(abs(t) for t in terms)
        err = abs(Fraction(float.fromhex(got)) - total)
        assert err <= Fraction(1, 2 ** 52) * abs(total) + Fraction(1, 2 ** 57) * size
