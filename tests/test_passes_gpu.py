"""The passes of a frame run side by side on the pixel schedule, each into a
buffer of its own, added in their order; the persistent schedule runs one after
the other.  Fewer passes than lanes, more (a lane taken again), one pixel, and
ragged frames; the diagnostics are the last pass's.

In FP64 the two schedules' kernels agree to the rounding of the float image (a
few ulp of the larger of the pixel and the frame's rms, 2^-20).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import AccretionDisc, Blackbody, Kerr  # noqa: E402


@pytest.mark.parametrize("samples", [2, 3])
@pytest.mark.parametrize("size", [(1, 1), (33, 19)])
def test_passes_side_by_side(built_lib, size, samples):
    cam = scene.Camera.look_at(scene.kerr_position(15.0, 80.0, 0.9), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
    with stg.Context(workloads.sky(128, 64), disc=AccretionDisc(3.0, 25.0, Blackbody(), 0.5)) as ctx:
        x, y = (ctx.render_raw(cam, Kerr(1.0, 0.9), ctx.params(
            _abi.ST_SEM_DRAFT, precision=_abi.ST_PREC_FP64, schedule=sched, width=size[0], height=size[1],
            samples=samples, pixel_jitter=1, exit_landing=1), diag=True)
            for sched in (_abi.ST_SCHED_PIXEL, _abi.ST_SCHED_PERSISTENT))
    for k in ("rays", "steps", "launches"):
        assert x.stats[k] == y.stats[k], k
    scale = np.maximum(np.abs(y.image), np.sqrt((y.image.astype(np.float64) ** 2).mean()))
    assert (np.abs(x.image - y.image) <= 2.0 ** -20 * scale).all()
    np.testing.assert_array_equal(x.diag["steps"], y.diag["steps"])
    np.testing.assert_array_equal(x.diag["flags"], y.diag["flags"])
