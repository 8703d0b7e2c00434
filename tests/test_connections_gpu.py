"""Connection rays (bidirectional, VCM, next-event estimation) stop at the first
hit that hides their target: images against the oracle, which finds the closest
hit, with a plate at all distances from the light around the tolerance at which
a hit counts as the target itself (1e-5), and the connections of both renderers
that make them."""
import numpy as np
import pytest

import wr_oracle
from walkray_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def plate_scene(gap):
    s = S.Scene("plate")
    s.add(S.MAT_DIFFUSE, *S.quad((-1, 0, -1), (-1, 0, 1), (1, 0, 1), (1, 0, -1), (0, 1, 0)), albedo=(0.7, 0.6, 0.5))
    s.add(S.MAT_EMISSIVE, *S.quad((-0.3, 1, -0.3), (0.3, 1, -0.3), (0.3, 1, 0.3), (-0.3, 1, 0.3), (0, -1, 0)),
          emission=(5.0, 4.0, 3.0))
    y = 1.0 - gap
    s.add(S.MAT_DIFFUSE, *S.quad((0.0, y, -0.4), (0.4, y, -0.4), (0.4, y, 0.4), (0.0, y, 0.4), (0, -1, 0)),
          albedo=(0.5, 0.5, 0.5))
    s.camera = S.Camera.from_fov((0, 0.6, -2.4), (0, 0.3, 0), (0, 1, 0), 29, 23, 50.0)
    return s


@pytest.mark.parametrize("gap", [0.5, 1e-2, 3e-4, 1e-4, 3e-5, 5e-6, 1e-6])
def test_connections_match_the_closest_hit(ctx, gap):
    s = plate_scene(gap)
    h, w = s.camera.height, s.camera.width
    sid, orc = ctx.upload(s), wr_oracle.SceneOracle(s)
    g = ctx.render(sid, 8, 3, seed=7, mode="bidirectional")
    o = orc.render_bpt(8, 3, seed=7)[0].reshape(h, w, 3) / 8
    assert np.isclose(g, o, rtol=1e-3, atol=1e-5).mean() > 0.99
    for mode in ("megakernel", "wavefront"):
        g = ctx.render(sid, 8, 3, seed=7, mode=mode, nee=True)
        o = orc.render(8, 3, seed=7, flags=wr_oracle.NEE)[0].reshape(h, w, 3) / 8
        assert np.isclose(g, o, rtol=1e-3, atol=1e-5).mean() > 0.99
    ctx.release(sid)
