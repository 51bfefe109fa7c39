"""The float-pair arithmetic of the FP64 frames (spacetime_gb300/csrc/st_df.cuh),
compiled for the host and measured against 128-bit arithmetic: the integration
(slopes in float pairs, state in three floats) is closer to the exact RK4
sequence than the same integration in double, and the shading functions keep
the 2^-36 that a float image needs with room to spare."""
import os
import platform
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def numbers(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("df") / "df_math")
    quad = ["-lquadmath"] if platform.machine() == "x86_64" else []
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "df_math.cpp")] + quad,
                   check=True)
    return [line.split() for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]


@pytest.mark.parametrize("row", range(4))
def test_integration_is_no_further_off_than_double(numbers, row):
    _, a, n, med_double, med_pairs, p90_double, p90_pairs = numbers[row]
    assert int(n) > 150
    assert float(med_pairs) <= float(med_double)
    assert float(p90_pairs) <= float(p90_double)


def test_shading_functions(numbers):
    _, e, _, lg, _, at = numbers[4]
    assert float(e) < 2.0 ** -36 and float(lg) < 2.0 ** -36 and float(at) < 2.0 ** -36
