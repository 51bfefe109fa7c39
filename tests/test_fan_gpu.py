"""The FP32 deflection fan (its own planar kernel) against the FP64 fan (the
general integrator) at the same camera radius: inside and outside the photon
sphere, near and far, with the last step landed on the escape sphere or not, and
at a step size whose budget ends rays.

Tolerance: an FP32 ray of N steps is off by at most N 2^-24 of its state (N up
to 4,000: 2.4e-4) and the exit angle grows as the inverse of the distance from
the critical angle; 20 coarse spacings (pi / 4095 each) from it that is a
factor of 65 on the angle: 1.6e-2 rad, for the linear worst case.  The
periapsis is off by the same fraction of itself.
"""
import math

import numpy as np
import pytest

from spacetime_gb300 import _abi, workloads
from spacetime_gb300.api import Context
from spacetime_gb300.scene import Camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("landing", [0, 1])
@pytest.mark.parametrize("r", [2.6, 3.0, 8.0, 30.0, 100.0])
def test_fp32_fan_matches_the_general_integrator(built_lib, r, landing):
    wl = workloads.config0().scaled(32, 18)
    cam = Camera.look_at((0.0, -r, 0.0), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), wl.cam.fov_factor)
    with Context(workloads.sky(64, 32), disc=None, emitter=wl.emitter) as ctx:
        fans = [ctx.sky_fan(cam, wl.bh, ctx.params(_abi.ST_SEM_DRAFT, width=32, height=18, precision=prec, samples=1,
                                                   pixel_jitter=0, exit_landing=landing))
                for prec in (_abi.ST_PREC_FP32, _abi.ST_PREC_FP64)]
    (a, fine, band), (b, _, band64) = fans
    a, b = a.astype(np.float64), b.astype(np.float64)
    k = np.arange(len(a))
    flips = np.nonzero(b[1:, 0] != b[:-1, 0])[0]
    assert flips.size == 1 and abs(np.nonzero(a[1:, 0] != a[:-1, 0])[0] - flips[0]).max() <= 1
    assert np.abs(band - band64).max() <= 1.01 * math.pi / 4095
    away = np.abs(k - flips[0]) > 20
    assert np.array_equal(a[away, 0], b[away, 0])
    esc = away & (b[:, 0] > 0.5)
    ang = np.abs(np.arctan2(a[esc, 1] * b[esc, 2] - a[esc, 2] * b[esc, 1], (a[esc, 1:3] * b[esc, 1:3]).sum(1)))
    assert ang.max() <= 1.6e-2, ang.max()
    assert (np.abs(a[esc, 3] - b[esc, 3]) <= 1.6e-2 * b[esc, 3]).all()
    # the fine fan spans the band and holds both outcomes
    assert 0.0 < fine[:, 0].mean() < 1.0 and np.isfinite(fine).all()
