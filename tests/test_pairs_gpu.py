"""FP64 frames on the pixel schedule integrate on the FP32 pipe
(spacetime_gb300/csrc/st_trace_pairs.cu); the persistent schedule keeps the
all-double kernels.  The two take the same steps and gas samples and give the
same image in every form the rule accepts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import AccretionDisc, Blackbody, Kerr, Schwarzschild  # noqa: E402


def _both(ctx, cam, bh, sem, **kw):
    out = []
    for sched in (_abi.ST_SCHED_PIXEL, _abi.ST_SCHED_PERSISTENT):
        p = ctx.params(sem, precision=_abi.ST_PREC_FP64, schedule=sched, **kw)
        out.append(ctx.render_raw(cam, bh, p))
    return out


def _same(a, b):
    """Same counts; every pixel within the float image's rounding (a few ulp of
    the larger of the pixel and the frame's rms, 2^-20)."""
    for k in ("rays", "steps", "gas_samples"):
        assert a.stats[k] == b.stats[k], (k, a.stats[k], b.stats[k])
    scale = np.maximum(np.abs(b.image), np.sqrt((b.image.astype(np.float64) ** 2).mean()))
    assert (np.abs(a.image - b.image) <= 2.0 ** -20 * scale).all()


@pytest.mark.parametrize("kind,a,M,size,kw", [
    ("gas", 0.9, 1.0, (50, 27), dict(exit_landing=1)),
    ("gas", 0.0, 1.0, (17, 9), dict(exit_landing=0, relativistic=1)),
    ("thick", 0.7, 1.0, (33, 19), dict(exit_landing=1)),          # rays become opaque inside a queue
    ("thick", 0.0, 1.0, (24, 13), dict(exit_landing=1, samples=2, pixel_jitter=1)),
    ("disc", 0.95, 1.0, (41, 23), dict(exit_landing=1, block_x=32, block_y=4)),
    ("disc", -0.5, 2.0, (16, 8), dict(exit_landing=0)),
    ("empty", 0.0, 0.5, (1, 1), dict(exit_landing=1)),
    ("empty", 0.3, 1.0, (37, 1), dict(exit_landing=1, dt=0.05, nmax=700)),
])
def test_draft_frames(built_lib, kind, a, M, size, kw):
    cam = scene.Camera.look_at(scene.kerr_position(15.0 * M, 80.0, a), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
    bh = Kerr(M, a) if a else Schwarzschild(M)
    disc = AccretionDisc(3.0 * M, 25.0 * M, Blackbody(), 0.5) if kind == "disc" else None
    vol = None
    if kind in ("gas", "thick"):
        vol = scene.make_volume(inner=2.32, outer=25.0, nr=48, nphi=24, nz=12, scale_height=0.05,
                                opacity_scale=1.2 if kind == "gas" else 60.0)
    with stg.Context(workloads.sky(128, 64), disc=disc, volume=vol) as ctx:
        a_, b_ = _both(ctx, cam, bh, _abi.ST_SEM_DRAFT, width=size[0], height=size[1],
                       **{"samples": 1, "pixel_jitter": 0, **kw})
    _same(a_, b_)


@pytest.mark.parametrize("size,emitter", [((31, 18), _abi.ST_EMIT_KEPLER), ((20, 11), _abi.ST_EMIT_KS_EXACT)])
def test_render_frames(built_lib, size, emitter):
    w = workloads.config0()
    with stg.Context(workloads.sky(128, 64), disc=w.disc, emitter=emitter) as ctx:
        a_, b_ = _both(ctx, w.cam, w.bh, _abi.ST_SEM_RENDER, width=size[0], height=size[1])
    _same(a_, b_)


def test_outside_the_rule_the_double_kernel_runs(built_lib):
    """A hole of 1e4 (lengths beyond the pair kernel's range) renders as before:
    the same frame as the persistent double kernel."""
    M = 1e4
    cam = scene.Camera.look_at((0.0, -15.0 * M, 2.0 * M), (0, 0, 0), (0, 0, 1), 0.75)
    with stg.Context(workloads.sky(128, 64)) as ctx:
        a_, b_ = _both(ctx, cam, Schwarzschild(M), _abi.ST_SEM_DRAFT, width=16, height=9, samples=1, pixel_jitter=0,
                       dt=0.05 * M, nmax=4000)
    _same(a_, b_)


def test_labels_do_not_depend_on_the_queue(built_lib):
    """Every row is written, whatever the set's size (below a warp, ragged, on
    either side of the warp-count rule) and the order its rays are taken in: a
    row has the same bits in every set that holds it."""
    from spacetime_gb300.surrogate import Surrogate
    s = Surrogate()
    big = s.generate(66001, offset=5)
    for n, off in ((1, 5), (31, 5), (33, 17), (1000, 60005), (65536, 5), (65537, 300)):
        for a_, b_ in zip(s.generate(n, offset=off), big):
            assert np.isfinite(a_).all() and np.array_equal(a_, b_[off - 5:off - 5 + n])
    s.close()
