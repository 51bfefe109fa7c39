"""The guard step of the guarded precisions (spacetime_gb300/csrc/st_df.cuh,
rk4_six and add_rn), compiled for the host: on the guarded state, two floats a
component, it is as exact as a step formed in double.  What a ray is off by is the
state's rounding, which both pay once a step.

Tolerance: a median over n rays of the same rounding noise scatters by about
1.25 / sqrt(n) of itself; the difference of two, at two deviations and n = 200: a
factor of 1.3.
"""
import os
import platform
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("df") / "df_guard")
    quad = ["-lquadmath"] if platform.machine() == "x86_64" else []
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "df_guard.cpp")] + quad,
                   check=True)
    return [line.split() for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]


@pytest.mark.parametrize("row", range(4))
def test_guard_step(rows, row):
    _, n, med_double, med_pairs = (float(x) for x in rows[row])
    assert n > 150
    assert med_pairs <= 1.3 * med_double
