"""The memory of the flights through heterogeneous media, 16 B for each path of
the queue, is taken when a scene with a density grid is first rendered."""
import pytest

from walkray_gb300 import scenes as S
from walkray_gb300.api import Context

pytestmark = pytest.mark.gpu


def test_flights_are_reserved_for_scenes_with_a_grid(built):
    import torch

    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    with Context() as c:
        plain, media = c.upload(S.cornell(32, 32)), c.upload(S.cornell_media(32, 32, grid_n=16))
        c.render(plain, 1, 8, mode="wavefront")
        before = free()
        c.render(media, 1, 8, mode="wavefront")
        assert before - free() >= 16 << 24
        after = free()
        c.render(plain, 1, 8, mode="wavefront")
        c.render(media, 1, 8, mode="wavefront")
        assert free() == after  # once
