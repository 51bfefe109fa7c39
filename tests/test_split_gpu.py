"""Small FP32 gas frames on the pixel schedule integrate and shade in separate
warps (spacetime_gb300/csrc/st_trace_split.cuh).  Against the kernel that marches
the gas between its steps: the pixel schedule's, through a track of one frame,
or the persistent schedule's where there are several passes.  Partial tiles, rays that end opaque inside a batch,
more samples than are evaluated together, budgets inside a batch, several
passes, and the largest frame of the rule.

The steps round alike.  A ray's image is a sum over at most 2,000 samples whose
last places may round otherwise (the compiler contracts them kernel by kernel),
2,000 x 2^-24 of the larger of the pixel and the frame's rms; an opacity that
crosses its threshold one sample later may cost a ray a few steps, 1e-4 of all.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import Kerr, Schwarzschild  # noqa: E402


@pytest.mark.parametrize("a,size,opacity,stride,kw", [
    (0.9, (1, 1), 1.2, 2, {}),
    (0.0, (9, 5), 1.2, 2, dict(relativistic=1)),
    (0.7, (33, 19), 60.0, 2, {}),                       # rays become opaque inside a batch
    (0.0, (24, 13), 60.0, 1, dict(samples=2, pixel_jitter=1)),
    (0.95, (40, 23), 1.2, 1, dict(dt=0.05)),            # several samples a step
    (0.3, (37, 3), 1.2, 2, dict(exit_landing=0, nmax=703)),
    (0.9, (256, 256), 6.0, 2, {}),
])
def test_split_frames(built_lib, a, size, opacity, stride, kw):
    cam = scene.Camera.look_at(scene.kerr_position(15.0, 80.0, a), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
    vol = scene.make_volume(inner=2.32, outer=25.0, nr=48, nphi=24, nz=12, scale_height=0.05, opacity_scale=opacity,
                            march_stride=stride)
    with stg.Context(workloads.sky(128, 64), disc=None, volume=vol) as ctx:
        bh = Kerr(1.0, a) if a else Schwarzschild(1.0)
        kw = {"samples": 1, "pixel_jitter": 0, "exit_landing": 1, **kw}
        px, ps = (ctx.params(_abi.ST_SEM_DRAFT, precision=_abi.ST_PREC_FP32, schedule=sched, width=size[0],
                             height=size[1], **kw) for sched in (_abi.ST_SCHED_PIXEL, _abi.ST_SCHED_PERSISTENT))
        x = ctx.render_raw(cam, bh, px)
        y = ctx.render_frames_raw([cam], bh, px) if kw["samples"] == 1 else ctx.render_raw(cam, bh, ps)
    y.image = y.image.reshape(x.image.shape)
    assert x.stats["rays"] == y.stats["rays"]
    for k in ("steps", "gas_samples"):
        assert y.stats[k] > 0 and abs(x.stats[k] - y.stats[k]) <= 1e-4 * y.stats[k], (k, x.stats[k], y.stats[k])
    scale = np.maximum(np.abs(y.image), np.sqrt((y.image.astype(np.float64) ** 2).mean()))
    assert (np.abs(x.image - y.image) <= 2000 * 2.0 ** -24 * scale).all()
