"""The FP32 fan's arithmetic.

- Its square root and its division by six (spacetime_gb300/csrc/st_round.cuh) are
  correctly rounded: every float from 2^-96 to 2^96 is compared.
- Its entries against the FP64 fan's at FP32's own level, so that a dropped term or a
  wrong landing in most of the fan would show.  A ray of N steps (4,000 at most) is
  off by at most N 2^-24, 2.4e-4, where bending does not magnify it, and bending
  magnifies it only near the critical angle: the median exit angle and the median
  periapsis are within that.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from spacetime_gb300 import _abi, workloads
from spacetime_gb300.api import Context, Schwarzschild
from spacetime_gb300.scene import Camera

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_roots_and_sixths_are_correctly_rounded(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "round_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-o", exe,
                    os.path.join(HERE, "round_check.cu")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "96"]


@pytest.mark.parametrize("M,r,kw", [(1.0, 3.0, {}), (1.0, 30.0, {}), (1.0, 30.0, dict(exit_landing=0)),
                                    (1.0, 100.0, {}), (0.1, 1.2, dict(dt=0.001)), (30.0, 600.0, dict(dt=0.6))])
def test_median_entry(built_lib, M, r, kw):
    cam = Camera.look_at((0.0, -r, 0.0), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 0.75)
    with Context(workloads.sky(64, 32), disc=None) as ctx:
        a, b = (ctx.sky_fan(cam, Schwarzschild(M), ctx.params(
            _abi.ST_SEM_DRAFT, width=32, height=18, precision=prec, samples=1, pixel_jitter=0,
            **{"exit_landing": 1, "dt": 0.02, **kw}))[0].astype(np.float64) for prec in (_abi.ST_PREC_FP32, _abi.ST_PREC_FP64))
    esc = (a[:, 0] > 0.5) & (b[:, 0] > 0.5)
    assert esc.sum() > 1000
    ang = np.abs(np.arctan2(a[esc, 1] * b[esc, 2] - a[esc, 2] * b[esc, 1], (a[esc, 1:3] * b[esc, 1:3]).sum(1)))
    assert np.median(ang) <= 4000 * 2.0 ** -24
    assert np.median(np.abs(a[esc, 3] / b[esc, 3] - 1.0)) <= 4000 * 2.0 ** -24
