"""The plain form's quotient by a reciprocal at hand (csrc/ionic_common.cuh)
against the division it stands for, at the edges of the range."""
import shutil
import struct
import subprocess
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
    double a, b;
    while (std::scanf("%la %la", &a, &b) == 2)
        std::printf("%la\n", cfg::cfg_quotient(a, b, 1.0 / b));
}
"""

NUMERATORS = [0.0, 1e-320, 1e-300, 3e-5, 1.0, 7.0 / 3.0, 1e17, 1e300, 1.7e308, np.inf, np.nan]
DIVISORS = [0.0, 1e-300, 3e-5, 1.0, 3.0, 1e17, 1e300, 1.7e308, np.inf, np.nan]


def _ordered(x):
    """Neighbouring doubles map to neighbouring integers."""
    i = struct.unpack("<q", struct.pack("<d", x))[0]
    return i if i >= 0 else -(2 ** 63) - i


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_quotient_is_the_division(tmp_path):
    """Infinite, zero and undefined quotients are the division's, the others
    within an ulp of it (the correction's rare ties and subnormal results)."""
    src, exe = tmp_path / "q.cpp", tmp_path / "q"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC), str(src), "-o",
                    str(exe)], check=True)
    pairs = [(s * a, t * b) for a in NUMERATORS for b in DIVISORS
             for s in (1.0, -1.0) for t in (1.0, -1.0)]
    text = "\n".join(f"{float(a).hex()} {float(b).hex()}" for a, b in pairs)
    out = subprocess.run([str(exe)], input=text, text=True, check=True,
                         capture_output=True).stdout.split()
    assert len(out) == len(pairs)
    with np.errstate(all="ignore"):
        for (a, b), got in zip(pairs, out):
            want, got = float(np.divide(a, b)), float.fromhex(got)
            if not np.isfinite(want) or want == 0.0:
                assert got == want or (np.isnan(got) and np.isnan(want)), (a, b, got, want)
            else:
                assert abs(_ordered(got) - _ordered(want)) <= 1, (a, b, got, want)
