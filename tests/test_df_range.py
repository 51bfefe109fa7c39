"""The gas shading's e^x of the FP64 frames (spacetime_gb300/csrc/st_df.cuh),
compiled for the host, at every argument that an optical depth can give it: the
user chooses opacity, spacing and density, so -x has no bound.

Tolerance: 2^-36 relative (as tests/test_df_math.py asks of the normal range)
down to -80; below, where the result's low half leaves a float's normal
exponents, one float rounding, 2^-23, and e^-87, where it ends.  A sample's emission
1 - e^x and the transmittance behind it stay in [0, 1].
"""
import math
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("df") / "df_exp_range")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "df_exp_range.cpp")], check=True)
    return exe


def test_exponential_of_any_optical_depth(harness):
    xs = [80.0, 1.0, 0.0, -1e-6, -0.3, -2.4, -39.9, -50.0, -79.0, -86.0, -86.99, -87.01, -88.0, -88.4, -88.9, -89.0,
          -96.0, -100.0, -104.0, -127.0, -500.0, -745.0, -1e4, -1e30, -math.inf]
    xs += [-80.0 - 0.37 * k for k in range(400)]
    out = subprocess.run([harness] + [repr(x) for x in xs], check=True, capture_output=True, text=True).stdout
    for x, line in zip(xs, out.splitlines(), strict=True):
        _, hi, lo, emission, through = map(float, line.split())
        want = math.exp(x)
        tol = 2.0 ** -36 * want if x >= -80.0 else 2.0 ** -23 * want + math.exp(-87.0)
        assert abs(hi + lo - want) <= tol, (x, hi, lo, want)
        if x <= 0.0:
            assert 0.0 <= emission <= 1.0 and 0.0 <= through <= 1.0, (x, emission, through)
