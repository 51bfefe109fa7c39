"""The fluid solver's grid barriers give up after a bounded number of polls.
SPACETIME_GB300_FLUID_WAIT=1 makes that one poll, so that blocks leave the launch
at its first barriers with nothing faulted and nothing hung.  A step that does not
wait cannot know; the next step and the next render do, and so do a timed step and
the solver's state.  The solver stays failed.  A new one on the same context, or a
volume set again, works as on a fresh context, to the same bits.
"""
import numpy as np
import pytest

from spacetime_gb300 import _abi, workloads
from spacetime_gb300.api import AccretionDisc, Blackbody, Context, DiscFluidSim
from spacetime_gb300.scene import make_volume

pytestmark = pytest.mark.gpu

W = workloads.config0().scaled(48, 27)


def _refused(f, *a, **kw):
    with pytest.raises(_abi.StError) as e:
        f(*a, **kw)
    assert e.value.code == _abi.ST_ECUDA


@pytest.mark.parametrize("nphi", [64, 256])   # the noise in blocks of its own, or as the advection goes
def test_a_barrier_that_runs_out(built_lib, monkeypatch, nphi):
    vol = make_volume(inner=3.0, outer=20.0, nr=96, nphi=nphi, nz=8, seed=5)
    disc = AccretionDisc(3.0, 20.0, Blackbody(wb_temperature=10000.0), 0.8)

    def params(ctx):
        return ctx.params(_abi.ST_SEM_DRAFT, width=48, height=27, precision=_abi.ST_PREC_FP32, samples=1, pixel_jitter=0)

    with Context(workloads.sky(64, 32), disc=disc, volume=vol) as ctx, DiscFluidSim(ctx, vol, disc) as sim:
        sim.step(dt=0.08, nsteps=3)
        want_state, want = sim.state(volume=True), ctx.render_raw(W.cam, W.bh, params(ctx)).image
    with Context(workloads.sky(64, 32), disc=disc, volume=vol) as ctx, DiscFluidSim(ctx, vol, disc) as sim:
        p = params(ctx)
        monkeypatch.setenv("SPACETIME_GB300_FLUID_WAIT", "1")
        sim.step(dt=0.08, nsteps=3)
        _refused(ctx.render_raw, W.cam, W.bh, p)       # the render waits for the steps before it
        monkeypatch.delenv("SPACETIME_GB300_FLUID_WAIT")
        _refused(sim.step, dt=0.08)
        _refused(sim.step, dt=0.08, timed=True)
        _refused(sim.state)
        _refused(ctx.render_frames_raw, [W.cam], W.bh, p)
        ctx.set_volume(vol)                             # the gas is whole, the solver is not
        ctx.render_raw(W.cam, W.bh, p)
        sim.step(dt=0.08)
        _refused(ctx.render_raw, W.cam, W.bh, p)
        ctx.set_volume(vol)
        with DiscFluidSim(ctx, vol, disc) as fresh:
            fresh.step(dt=0.08, nsteps=3)
            got_state, got = fresh.state(volume=True), ctx.render_raw(W.cam, W.bh, p).image
    for k in ("vu", "vv", "dens", "volume"):
        np.testing.assert_array_equal(got_state[k], want_state[k])
    np.testing.assert_array_equal(got, want)
