"""The low-variance estimators in the wavefront's finish kernel (its light
connections and the accumulators that the bounce loop hands over) against the
megakernel, which makes the same draws: with the loop run to its end, with the
last paths finished outside it, and with every path finished there from the
start.  Sums and sums of squares, so that each sample counts."""
import numpy as np
import pytest

import make_golden
from walkray_gb300.api import LOW_VARIANCE, Context

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def own(built):
    with Context() as c:
        yield c


@pytest.mark.parametrize("capacity,drain", [(1 << 14, 0), (1 << 14, 1 << 12), (1 << 14, 1 << 20), (1 << 24, -1),
                                            (1 << 24, 1 << 24)])
@pytest.mark.parametrize("name", ["mixed_l2", "cornell", "fog", "hetero"])
def test_finish_equals_the_megakernel(own, name, capacity, drain):
    sid = own.upload(make_golden.golden_scenes()[name])
    a1, a2 = own.render_stats(sid, 16, 16, seed=9, mode="megakernel", flags=LOW_VARIANCE)
    own.set_wavefront_config(capacity=capacity, drain_paths=drain)
    b1, b2 = own.render_stats(sid, 16, 16, seed=9, mode="wavefront", flags=LOW_VARIANCE)
    own.release(sid)
    assert np.allclose(a1, b1, rtol=1e-4, atol=1e-4), np.abs(a1 - b1).max()
    assert np.allclose(a2, b2, rtol=1e-3, atol=1e-3), np.abs(a2 - b2).max()
