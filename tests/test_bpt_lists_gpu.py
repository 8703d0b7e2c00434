"""The bidirectional renderer's connection lists, one per pair of light and eye
length, against the oracle's connections of the same sub-paths: sample counts
at and around a warp and a block, empty lists between full ones, the shortest
and the longest sub-paths (2 and 32 records).  Both sides compute the same
connections in the same precision; they differ by the order of the film's FP32
additions and by the last bits of powf (1e-3, as the paired tests)."""
import numpy as np
import pytest

import wr_oracle
from walkray_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,depth", [(1, 1, 8), (31, 1, 8), (33, 1, 8), (129, 1, 0), (37, 29, 30)])
def test_connection_lists_match_the_oracle(ctx, width, height, depth):
    s = S.cornell(width, height)
    sid = ctx.upload(s)
    g = ctx.render(sid, 8, depth, seed=71, mode="bidirectional").astype(np.float64)
    ctx.release(sid)
    o = wr_oracle.SceneOracle(s).render_bpt(8, depth, seed=71)[0].reshape(height, width, 3) / 8
    assert np.isclose(g, o, rtol=1e-3, atol=1e-5).mean() > 0.99
