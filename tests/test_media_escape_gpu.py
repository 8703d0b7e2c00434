"""A path inside an object that its ray leaves without a hit (an open mesh)
ends there: no object is looked up for the missing hit."""
import numpy as np
import pytest

from walkray_gb300 import scenes as S

pytestmark = pytest.mark.gpu

OPEN = {
    "homogeneous": dict(material=S.MAT_HOMOGENEOUS, sigma_s=(0.1, 0.1, 0.1), sigma_a=(0.1, 0.1, 0.1), g=0.1, ior=1.0),
    "heterogeneous": dict(material=S.MAT_HETEROGENEOUS, sigma_s=(0.8, 0.8, 0.8), sigma_a=(0.2, 0.2, 0.2), g=0.3,
                          ior=1.0, density_scale=1.0, step_size=0.01, grid_index=0),
    "refractive": dict(material=S.MAT_REFRACTIVE, ior=1.5),
}


@pytest.mark.parametrize("kind", sorted(OPEN))
@pytest.mark.parametrize("mode", ["megakernel", "wavefront"])
@pytest.mark.parametrize("nee", [False, True])
def test_a_path_that_leaves_an_open_object_ends(ctx, kind, mode, nee):
    s = S.Scene("open_" + kind)
    d = dict(OPEN[kind])
    if kind == "heterogeneous":
        s.grids.append(S.Grid(S.fbm_grid(8, 2, 1), (-1.0, -1.0, 0.0), (1.0, 1.0, 1.0)))
    s.add(d.pop("material"), [(-9, -9, 0), (9, -9, 0), (9, 9, 0), (-9, 9, 0)], [(0, 1, 2), (0, 2, 3)], **d)
    s.add(S.MAT_EMISSIVE, [(30, 0, 30), (30, 1, 30), (30, 0, 31)], [(0, 1, 2)], emission=(1.0, 1.0, 1.0))
    s.camera = S.Camera.from_fov((0, 0, -3), (0, 0, 0), (0, 1, 0), 37, 29, 40.0)
    sid = ctx.upload(s)
    img = ctx.render(sid, 2, 8, seed=1, mode=mode, nee=nee)
    ctx.release(sid)
    assert np.isfinite(img).all()
    if not nee:  # nothing here reaches the emitter
        assert (img == 0).all()
