"""Routes through the dispatch that other tests do not reach.

- FP64 tracks on pixel tiles (the pair kernel with a table of cameras, each with
  its own escape radius and step budget), captured or not, against the all-double
  kernels of the persistent schedule; a track with one frame beyond the pair
  kernel's range is all double.
- FP64 with the surrogate (the pair kernel over a list of pixels): pixels that the
  network does not serve are the plain frame's, bit for bit.
- The blackbody table in shared memory with gas: frames large enough for the kernel
  that stages it.
- Guard steps along the whole ray against FP64.  The guarded state is 48 bits and
  the step as exact as a double one; what is left is the photon energy, a float:
  2^-24 of it, and at most twice that in the exit direction of a median ray, 2^-23.
  Plain FP32 steps, 1,100 roundings of 2^-24 and their growth, are beyond that.
- Fluid steps in one call or in several (the `graph` argument selects nothing).
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import AccretionDisc, Blackbody, DiscFluidSim, Kerr, Schwarzschild  # noqa: E402

from .helpers import angle, gpu_render  # noqa: E402


def _near(x, y):
    scale = np.maximum(np.abs(y), np.sqrt((y.astype(np.float64) ** 2).mean()))
    assert (np.abs(x - y) <= 2.0 ** -20 * scale).all()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("kind,a,size,radii,pairs", [
    ("disc", 0.9, (33, 19), (15.0, 18.0, 27.0), True),
    ("gas", 0.9, (20, 11), (15.0, 40.0), True),
    ("gas", 0.0, (17, 9), (12.0, 12.5, 13.0), True),
    ("disc", 0.0, (16, 8), (15.0, 9e4), False),          # the second frame escapes at 1.8e5
])
def test_fp64_tracks_on_pixel_tiles(built_lib, kind, a, size, radii, pairs, graph):
    cams = [scene.Camera.look_at(scene.kerr_position(r, 80.0, a), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
            for r in radii]
    disc = AccretionDisc(3.0, 25.0, Blackbody(), 0.5) if kind == "disc" else None
    vol = scene.make_volume(inner=2.32, outer=25.0, nr=48, nphi=24, nz=12, scale_height=0.05) if kind == "gas" else None
    with stg.Context(workloads.sky(128, 64), disc=disc, volume=vol) as ctx:
        out = []
        for sched in (_abi.ST_SCHED_PIXEL, _abi.ST_SCHED_PERSISTENT):
            p = ctx.params(_abi.ST_SEM_DRAFT, precision=_abi.ST_PREC_FP64, schedule=sched, width=size[0],
                           height=size[1], samples=1, pixel_jitter=0, exit_landing=1, graph=graph)
            ctx.render_frames_raw(cams[::-1], Kerr(1.0, a) if a else Schwarzschild(1.0), p)
            out.append(ctx.render_frames_raw(cams, Kerr(1.0, a) if a else Schwarzschild(1.0), p))
    x, y = out
    for k in ("rays", "steps", "gas_samples"):
        assert x.stats[k] == y.stats[k], (k, x.stats[k], y.stats[k])
    for f in range(len(cams)):
        _near(x.image[f], y.image[f])
    if not pairs:
        np.testing.assert_array_equal(x.image, y.image)


def test_fp64_frame_with_the_surrogate(built_lib):
    from spacetime_gb300.surrogate import load_trained
    w = workloads.config1_thin().scaled(192, 108)
    sur = load_trained()
    with stg.Context(workloads.sky(512, 256), disc=None, emitter=w.emitter) as ctx:
        ctx.set_surrogate(sur)
        kw = dict(width=192, height=108, precision=_abi.ST_PREC_FP64, samples=1, pixel_jitter=0, exit_landing=1)
        a = ctx.render_raw(w.cam, w.bh, ctx.params(w.semantics, **kw), diag=True)
        b = ctx.render_raw(w.cam, w.bh, ctx.params(w.semantics, surrogate=1, surrogate_sigma=4e-4, **kw), diag=True)
    served = (b.diag["flags"] & _abi.ST_RAY_SURROGATE) > 0
    assert 0.2 < served.mean() < 0.8 and b.stats["surrogate_rays"] == served.sum()
    np.testing.assert_array_equal(a.image[~served], b.image[~served])
    np.testing.assert_array_equal(a.diag["steps"][~served], b.diag["steps"][~served])
    assert b.stats["steps"] == a.diag["steps"][~served].sum()
    sur.close()


def test_blackbody_table_in_shared_memory_with_gas(built_lib, monkeypatch):
    w = workloads.config1().scaled(320, 180)
    sky = workloads.sky(128, 64)
    a = gpu_render(w, sky, _abi.ST_PREC_FP32, diag=False)
    monkeypatch.setenv("SPACETIME_GB300_LUT_SMEM", "1")
    b = gpu_render(w, sky, _abi.ST_PREC_FP32, diag=False)
    monkeypatch.delenv("SPACETIME_GB300_LUT_SMEM")
    assert a.stats["gas_samples"] == b.stats["gas_samples"] > 0
    np.testing.assert_array_equal(a.image, b.image)


@pytest.mark.parametrize("prec", [_abi.ST_PREC_FP32_GUARDED, _abi.ST_PREC_FP32_GUARDED_DF])
@pytest.mark.parametrize("sched", [_abi.ST_SCHED_PIXEL, _abi.ST_SCHED_PERSISTENT])
@pytest.mark.parametrize("a", [0.9, 0.0])
def test_guard_steps_along_the_whole_ray(built_lib, a, sched, prec):
    w = dataclasses.replace(workloads.config1_thin().scaled(96, 54), disc=None)
    w.bh = Kerr(1.0, a) if a else Schwarzschild(1.0)
    w.params = dict(samples=1, pixel_jitter=0, exit_landing=1)
    sky = workloads.sky(128, 64)
    ref = gpu_render(w, sky, _abi.ST_PREC_FP64, schedule=_abi.ST_SCHED_PERSISTENT)
    guarded = gpu_render(w, sky, prec, schedule=sched, r_guard=1e3, renorm_every=64)
    plain = gpu_render(w, sky, _abi.ST_PREC_FP32)
    esc = lambda r: (r.diag["flags"] & _abi.ST_RAY_ESCAPED) > 0
    both = esc(ref) & esc(guarded) & esc(plain)
    assert both.mean() > 0.5
    # rays proven captured at launch take no guard steps
    free = (ref.diag["flags"] & _abi.ST_RAY_BCAPT) == 0
    assert (guarded.diag["fp64_steps"] == guarded.diag["steps"])[free].all()
    d, d32 = (np.median(angle(r.diag["dir"][both], ref.diag["dir"][both])) for r in (guarded, plain))
    assert d <= 2.0 ** -23 < d32, (d, d32)


@pytest.mark.parametrize("split", [(12,), (1, 11), (5, 1, 6)])
def test_fluid_steps_in_one_call_or_several(built_lib, split):
    vol = scene.make_volume(inner=3.0, outer=20.0, nr=96, nphi=128, nz=16, seed=5)
    disc = AccretionDisc(3.0, 20.0, Blackbody(wb_temperature=10000.0), 0.8)
    with stg.Context(workloads.sky(64, 32), disc=disc, volume=vol) as ctx, DiscFluidSim(ctx, vol, disc) as a, \
            DiscFluidSim(ctx, vol, disc) as b:
        a.step(dt=0.08, nsteps=12)
        want = a.state(volume=True)
        for k, n in enumerate(split):
            b.step(dt=0.08, nsteps=n, graph=bool(k % 2))
        got = b.state(volume=True)
    for k in ("vu", "vv", "dens", "volume"):
        np.testing.assert_array_equal(got[k], want[k])
    assert got["t"] == want["t"]
