"""FP64 gas frames on the pixel schedule (float-pair shading) against the
all-double kernels of the persistent schedule where one sample is optically
thick: an optical depth of opacity x density x march_stride x dt has no upper
bound, e^-tau falls out of a float's range at 88 and out of a double's at 745.
A gas that emits without absorbing, or amplifies (negative opacity), too.

Tolerance: the float image's rounding, as tests/test_pairs_gpu.py."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import Kerr, Schwarzschild  # noqa: E402


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("a,tau", [(0.9, 50.0), (0.0, 87.0), (0.9, 89.0), (0.0, 100.0), (0.9, 500.0), (0.5, 1e4),
                                   (0.9, 1e37), (0.0, 0.0), (0.9, -0.02)])
def test_optical_depth_of_a_sample(built_lib, a, tau, uniform):
    dt, stride = 0.02, 2
    vol = scene.make_volume(inner=2.32, outer=25.0, nr=48, nphi=24, nz=12, scale_height=0.05, march_stride=stride,
                            opacity_scale=tau / (stride * dt))
    if uniform:  # every sample has this optical depth
        vol = dataclasses.replace(vol, density=np.ones_like(vol.density))
    cam = scene.Camera.look_at(scene.kerr_position(15.0, 70.0, a), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
    with stg.Context(workloads.sky(128, 64), disc=None, volume=vol) as ctx:
        x, y = (ctx.render_raw(cam, Kerr(1.0, a) if a else Schwarzschild(1.0),
                               ctx.params(_abi.ST_SEM_DRAFT, precision=_abi.ST_PREC_FP64, schedule=sched, width=31,
                                          height=18, dt=dt, samples=1, pixel_jitter=0, exit_landing=1))
                for sched in (_abi.ST_SCHED_PIXEL, _abi.ST_SCHED_PERSISTENT))
    assert np.isfinite(y.image).all() and y.stats["gas_samples"] > 0
    for k in ("rays", "steps", "gas_samples"):
        assert x.stats[k] == y.stats[k], (k, x.stats[k], y.stats[k])
    scale = np.maximum(np.abs(y.image), np.sqrt((y.image.astype(np.float64) ** 2).mean()))
    assert (np.abs(x.image - y.image) <= 2.0 ** -20 * scale).all()
