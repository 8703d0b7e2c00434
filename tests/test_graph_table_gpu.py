"""The wavefront's captured bounce loops are kept per set of kernels: calls that
need different sets in turn (scenes with and without media, estimators with and
without light connections) take no longer than the same calls one kind at a time
(a capture on each call made them 1.5 to 1.6 times as long), and their images
stay the same."""
import time

import numpy as np
import pytest

from walkray_gb300 import scenes as S
from walkray_gb300.api import LOW_VARIANCE, Context

pytestmark = pytest.mark.gpu

CALLS = [("cornell", 0), ("media", 0), ("cornell", LOW_VARIANCE), ("media", LOW_VARIANCE)]


@pytest.fixture(scope="module")
def alternating(built):
    """A context whose calls all run the bounce loop, with a scene of each kind."""
    with Context() as c:
        c.set_wavefront_config(capacity=1 << 14, drain_paths=0, iters_per_graph=1)
        sids = {"cornell": c.upload(S.cornell(8, 8)), "media": c.upload(S.cornell_media(8, 8, grid_n=16))}
        yield lambda k, depth: c.render(sids[CALLS[k][0]], 1, depth, seed=3, mode="wavefront", flags=CALLS[k][1])


def microseconds(call):
    t = time.perf_counter()
    call()
    return (time.perf_counter() - t) * 1e6


@pytest.mark.parametrize("first,second", [(0, 1), (0, 2), (1, 3), (2, 3)])
def test_calls_in_turn_take_as_long_as_alone(alternating, first, second):
    alone, turn = [], []
    for k in (first, second):
        times = [microseconds(lambda: alternating(k, 1)) for _ in range(40)]
        alone.append(np.median(times[8:]))
    for _ in range(40):
        turn.append([microseconds(lambda: alternating(k, 1)) for k in (first, second)])
    turn = np.median(np.array(turn)[8:], axis=0)
    assert turn.sum() < 1.25 * sum(alone), (alone, turn)


def test_images_do_not_depend_on_the_calls_before(alternating):
    want = [alternating(k, 8) for k in range(len(CALLS))]
    for k in (0, 1, 0, 2, 3, 1, 2, 0, 3):
        # one path per pixel: added to the film once, so the same bits each time
        assert np.array_equal(alternating(k, 8), want[k])
