"""The guard step of the guarded precisions component by component
(spacetime_gb300/csrc/st_df.cuh, rk4_six), compiled for the host: the same sums and
products as the packed form of the FP64 frames' step, so the same bits."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_component_form_is_the_packed_one_bit_for_bit(tmp_path):
    exe = str(tmp_path / "df_six")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "df_six.cpp")],
                   check=True)
    rows = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(rows) == 4
    for row in rows:
        _, steps, differ = row.split()
        assert int(steps) > 10_000 and int(differ) == 0, row
