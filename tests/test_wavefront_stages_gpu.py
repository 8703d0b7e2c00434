"""The wavefront renderer's flights through heterogeneous media (k_wf_track) and
its finish of the last paths (k_wf_finish) against the megakernel, which walks
each path on one thread with the same draws: path counts at and around a warp,
a block and the lanes' refill, with the bounce loop run to the end and with all
paths finished outside it.  At one sample per pixel each pixel is one path, so
only the rounding of the kernels' own fused operations may differ (24 vertices
of some 20 operations at 2^-24 each: 3e-5)."""
import numpy as np
import pytest

from walkray_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drain", [0, 1 << 20])
@pytest.mark.parametrize("nee", [False, True])
@pytest.mark.parametrize("width,height", [(1, 1), (31, 1), (33, 1), (1, 129), (67, 61), (200, 153)])
def test_stages_equal_the_megakernel(ctx, width, height, nee, drain):
    sid = ctx.upload(S.cornell_media(width, height, grid_n=16, seed=3))
    a = ctx.render(sid, 1, 24, seed=5, mode="megakernel", nee=nee)
    try:
        ctx.set_wavefront_config(capacity=1 << 14, drain_paths=drain)
        b = ctx.render(sid, 1, 24, seed=5, mode="wavefront", nee=nee)
    finally:
        ctx.set_wavefront_config(capacity=1 << 24)
    ctx.release(sid)
    assert np.allclose(a, b, rtol=1e-4, atol=1e-5), np.abs(a - b).max()


@pytest.mark.parametrize("width,height", [(1023, 1), (32, 32), (41, 25), (64, 48)])
def test_sorted_paths_equal_the_megakernel(ctx, width, height):
    """Path counts at and around the sort stage's tile of 1024, materials mixed."""
    s = S.mixed_spheres(width, height, seed=7, level=2)
    sid = ctx.upload(s)
    a = ctx.render(sid, 1, 16, seed=3, mode="megakernel")
    try:
        ctx.set_wavefront_config(capacity=1 << 14, drain_paths=0)
        b = ctx.render(sid, 1, 16, seed=3, mode="wavefront")
    finally:
        ctx.set_wavefront_config(capacity=1 << 24)
    ctx.release(sid)
    assert np.allclose(a, b, rtol=1e-4, atol=1e-5), np.abs(a - b).max()
