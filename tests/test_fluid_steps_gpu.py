"""The one-launch fluid steps at the edges of their tiling and scheduling: grids
smaller than a tile or a halo (which then wraps around the disc more than
once), ragged ones, more tiles than SMs, enough for launches by phase, and sweep
counts at and beyond one pass.  Without transcendental functions (drag 0, relax 0) the state equals the
oracle's bit for bit; steps in one call or several give the same bits.
"""
import numpy as np
import pytest

from oracle import oracle as O
from spacetime_gb300 import workloads
from spacetime_gb300.api import AccretionDisc, Blackbody, Context, DiscFluidSim
from spacetime_gb300.scene import make_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jacobi", [2, 16, 17])
@pytest.mark.parametrize("nr,nphi,nz", [(2, 1, 2), (33, 7, 3), (31, 130, 9), (700, 100, 2), (1000, 130, 2)])
def test_bits_at_the_edges(built_lib, nr, nphi, nz, jacobi):
    vol = make_volume(inner=3.0, outer=20.0, nr=nr, nphi=nphi, nz=nz, seed=5)
    disc = AccretionDisc(3.0, 20.0, Blackbody(wb_temperature=10000.0), 0.8)
    kw = dict(drag=0.0, relax=0.0)
    orc = O.FluidSim(vol, 3.0, 20.0, falloff=0.8, **kw)
    orc.step(dt=0.08, jacobi=jacobi, nsteps=4)
    with Context(workloads.sky(64, 32), disc=disc, volume=vol) as ctx, DiscFluidSim(ctx, vol, disc, **kw) as one, \
            DiscFluidSim(ctx, vol, disc, **kw) as several:
        for n in (1, 2, 1):
            several.step(dt=0.08, jacobi=jacobi, nsteps=n)
        b = several.state(volume=True)
        one.step(dt=0.08, jacobi=jacobi, nsteps=4)
        a = one.state(volume=True)
    assert a["t"] == b["t"] == orc.t
    for k in ("vu", "vv", "dens"):
        np.testing.assert_array_equal(a[k], getattr(orc, k), err_msg=k)
        np.testing.assert_array_equal(b[k], a[k], err_msg=k)
    np.testing.assert_array_equal(a["volume"], a["dens"][None] * orc.env[:, None, :])
    np.testing.assert_array_equal(b["volume"], a["volume"])
