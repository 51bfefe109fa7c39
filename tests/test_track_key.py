"""A captured camera track is replayed as long as its launch block is the same: the
block may hold sizes and rules, nothing that moves with the cameras.  Of the
frames' escape radii it keeps one bit, the range of the FP64 pair kernel."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs the CUDA headers")
def test_launch_block_of_a_track(tmp_path):
    exe = str(tmp_path / "track_key")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(NVCC))), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", inc, "-o", exe, os.path.join(HERE, "track_key.cpp")], check=True)
    out = subprocess.run([exe, "30", "31", "60", "9e4", "30", "2e5", "2e5", "3e5", "99999", "100001"], check=True,
                         capture_output=True, text=True).stdout.split()
    rows = [tuple(map(int, out[k:k + 3])) for k in range(0, len(out), 3)]
    assert rows == [(1, 1, 1), (1, 1, 1), (0, 1, 0), (1, 0, 0), (1, 0, 0)]
