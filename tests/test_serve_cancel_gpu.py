"""Paths of a cancelled request that are still inside a heterogeneous medium end
while other requests, with media and without, run on: every request reaches its
final state."""
import time

import numpy as np
import pytest

from walkray_gb300 import scenes as S
from walkray_gb300.api import Context, Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", ["fog", "cornell"])
def test_cancelled_media_request_drains(built, other):
    ctx = Context()
    media = ctx.upload(S.cornell_media(32, 32, grid_n=16, seed=3))
    rest = ctx.upload(S.cornell_fog(32, 32) if other == "fog" else S.cornell(32, 32))
    srv = Server(ctx)
    try:
        long = srv.submit(rest, 128, 128, 2048, 24, seed=2)
        for k in range(4):
            big = srv.submit(media, 128, 128, 4096, 24, seed=3 + k)
            time.sleep(0.02)
            srv.cancel(big)
            st = srv.wait([big], timeout=60)
            assert st[big]["state"] == "cancelled"
        st = srv.wait([long], timeout=120)
        assert st[long]["state"] == "done"
        img = srv.fetch(long)
    finally:
        srv.stop()
    assert np.isfinite(img).all() and img.mean() > 0
    ctx.close()
