"""Frames of several passes where device memory is short.  The buffers of the
passes beside the first are an extra: without the memory for them a frame renders
with fewer side by side, to the same bits, and buffers that an earlier frame left
in the context are given up when a later call needs the memory.

The rest of the GPU's memory is held by one allocation meanwhile, all but some
frames' worth.
"""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

import spacetime_gb300 as stg  # noqa: E402
from spacetime_gb300 import _abi, scene, workloads  # noqa: E402
from spacetime_gb300.api import AccretionDisc, Blackbody, Kerr  # noqa: E402

N = 2048                    # a side; a frame buffer is 64 MiB, three of them 192
FRAME = N * N * 16
CAM = scene.Camera.look_at(scene.kerr_position(15.0, 80.0, 0.9), (0, 0, 0), (0, 0, 1), scene.lens_fov(24.0))
BH = Kerr(1.0, 0.9)


def _ctx():
    return stg.Context(workloads.sky(128, 64), disc=AccretionDisc(3.0, 25.0, Blackbody(), 0.5))


def _params(ctx, **kw):
    return ctx.params(_abi.ST_SEM_DRAFT, precision=_abi.ST_PREC_FP32, width=N, height=N, exit_landing=1,
                      **{"samples": 1, "pixel_jitter": 0, **kw})


@contextlib.contextmanager
def _hold_all_but(nbytes):
    torch = pytest.importorskip("torch")
    torch.cuda.empty_cache()
    try:
        held = torch.empty(torch.cuda.mem_get_info()[0] - nbytes, dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pytest.skip("the GPU's memory is not free in one piece")
    try:
        free = torch.cuda.mem_get_info()[0]
        if not 0.8 * nbytes <= free <= 1.1 * nbytes:
            pytest.skip(f"{free} bytes left of {nbytes} asked for")
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_a_frame_of_several_passes_needs_no_extra_memory(built_lib):
    with _ctx() as ctx:
        want = ctx.render_raw(CAM, BH, _params(ctx, samples=2, pixel_jitter=1))
    with _ctx() as ctx:
        ctx.render_raw(CAM, BH, _params(ctx))   # the frame's own buffers
        with _hold_all_but(FRAME + FRAME // 2):
            got = ctx.render_raw(CAM, BH, _params(ctx, samples=2, pixel_jitter=1))
    assert got.stats["status"] == _abi.ST_OK
    for k in ("rays", "steps", "launches"):
        assert got.stats[k] == want.stats[k], k
    np.testing.assert_array_equal(got.image, want.image)


def test_pass_buffers_are_given_up(built_lib):
    with _ctx() as ctx:
        want = ctx.render_depth_raw(CAM, BH, _params(ctx), nbuckets=4)   # buckets: 192 MiB
    with _ctx() as ctx:
        ctx.render_raw(CAM, BH, _params(ctx, samples=2, pixel_jitter=1))
        with _hold_all_but(FRAME + FRAME // 2):
            got = ctx.render_depth_raw(CAM, BH, _params(ctx), nbuckets=4)
    np.testing.assert_array_equal(got.image, want.image)
