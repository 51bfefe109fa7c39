"""Small FP32 gas frames (spacetime_gb300/csrc/st_trace_split.cuh) at the edges of
their rule and of their batches: the largest frame that it takes and the first
that it leaves, and step budgets that end inside and at the ends of the first
batches (of 16 steps), against the kernel that marches the gas between its steps,
through a track of one frame.  Tolerance: as
tests/test_split_gpu.py derives it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import Kerr, Schwarzschild  # noqa: E402


@pytest.mark.parametrize("a,size,opacity,kw", [
    (0.9, (192, 128), 1.2, {}),
    (0.0, (193, 128), 1.2, {}),
    *[(0.0 if n % 2 else 0.9, (13, 7), 1.2 if n % 3 else 3000.0, dict(nmax=n)) for n in
      (1, 2, 15, 16, 17, 31, 32, 33, 48)],
    (0.9, (40, 30), 3000.0, {}),                        # rays end in the gas within a few steps
    (0.998, (21, 17), 1.2, {}),                         # a spin that the rule leaves
])
def test_split_edges(built_lib, a, size, opacity, kw):
    # inside the slab, so that the first steps have samples
    cam = scene.Camera.look_at(scene.kerr_position(15.0, 88.0, a), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
    vol = scene.make_volume(inner=2.32, outer=25.0, nr=48, nphi=24, nz=12, scale_height=0.1, opacity_scale=opacity,
                            march_stride=1)
    with stg.Context(workloads.sky(128, 64), disc=None, volume=vol) as ctx:
        bh = Kerr(1.0, a) if a else Schwarzschild(1.0)
        p = ctx.params(_abi.ST_SEM_DRAFT, precision=_abi.ST_PREC_FP32, width=size[0], height=size[1], samples=1,
                       pixel_jitter=0, exit_landing=1, **kw)
        x = ctx.render_raw(cam, bh, p)
        y = ctx.render_frames_raw([cam], bh, p)
    y.image = y.image.reshape(x.image.shape)
    assert x.stats["rays"] == y.stats["rays"] and y.stats["gas_samples"] > 0
    for k in ("steps", "gas_samples"):
        assert abs(x.stats[k] - y.stats[k]) <= 1e-4 * y.stats[k], (k, x.stats[k], y.stats[k])
    scale = np.maximum(np.abs(y.image), np.sqrt((y.image.astype(np.float64) ** 2).mean()))
    assert (np.abs(x.image - y.image) <= 2000 * 2.0 ** -24 * scale).all()
