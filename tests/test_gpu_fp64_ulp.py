"""MathF64's reciprocals, quotients and roots (emma_b200/csrc/hydro_math.cuh) one by one,
in units of the last place, against CUDA's 1 / b, a / b and sqrt, and the fifth roots
against the host's long double power (tests/fp64_math_check.cu)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

# (largest difference, largest share of pairs that differ).  A result whose value before the
# last rounding is off by a relative 2^-k changes that rounding with probability below
# 2^(54 - k): rcp 2^-80 and root2 2^-78 from 20-bit seeds, 1.5e-8 and 6e-8; a twelfth of the
# divisors and half of the roots are chosen where that is likelier: a factor of four.  The
# reciprocal of an all-ones mantissa lies 2^-106 above a boundary, and may round either way.
# div_y is exact for a correctly rounded reciprocal, over_g1 everywhere; div_yy's reciprocal
# is within an ulp, its quotient off within 2^-105 of a boundary.
BOUNDS = {
    "rcp": (1, 6e-8),
    "rcp_ones": (1, 1.0),
    "root2": (1, 2.4e-7),
    "quot": (1, 6e-8),
    "quot_ones": (1, 1.0),
    "div_y": (0, 0.0),
    "div_yy": (1, 6e-8),
    "over_g1": (0, 0.0),
    # 0.5 and what the estimate of ln x and the products' roundings add, 0.01
    "root5": (0.51, 0.01),
    "root5_rcp": (0.51, 0.01),
    "root5_near": (0.51, 0.01),
}


def test_fp64_functions_in_ulp(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fp64_math_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    os.path.join(HERE, "fp64_math_check.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    got = {w[0]: (float(w[3]), float(w[2]) / float(w[1])) for w in (line.split() for line in out.splitlines())}
    assert set(got) == set(BOUNDS), out
    for name, (ulp, share) in BOUNDS.items():
        assert got[name][0] <= ulp and got[name][1] <= share, out
