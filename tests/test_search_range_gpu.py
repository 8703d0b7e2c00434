"""The four-wide search over the whole range of directions and coordinates that
it takes (wr_quad.cuh: |d| from 1e-15 to 1e14, coordinates to 1e15 |d|) against the
walk that visits every box the reference visits: the same triangle ids and the
same t bit for bit on both sides of the range's ends, and rays of any length at
the speed of unit ones."""
import numpy as np
import pytest

from test_search_gpu import pair, rays_of, same_hits, scene_of, soup  # noqa: F401  (pair: a fixture)
from walkray_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-16, -15, -14, -8, -6, -3, 3, 6, 8, 14, 15, 16, 20])
@pytest.mark.parametrize("scene", ["mixed", "grid", "overlap"])
def test_directions_of_any_length(pair, scene, exponent):  # noqa: F811
    s = scene_of(scene)
    r = rays_of(s, "corners", 20000)
    rng = np.random.default_rng(exponent + 100)
    r[:, 3:] *= (10.0 ** (exponent + rng.uniform(-0.5, 0.5, (len(r), 1)))).astype(np.float32)
    same_hits(pair, s, r)


@pytest.mark.parametrize("size", [1e-20, 1e-6, 1e6, 1e12, 1e17, 1e18, 1e19])
@pytest.mark.parametrize("kind", ["plain", "axis", "scaled"])
def test_scenes_of_any_size(pair, size, kind):  # noqa: F811
    v, f = soup(500, np.random.default_rng(3), 0.5)
    s = S.Scene("sized")
    s.add(S.MAT_DIFFUSE, (v * size).astype(np.float32), f)
    same_hits(pair, s, rays_of(s, kind, 20000))


def test_hits_at_an_infinite_distance(pair):  # noqa: F811
    """Slivers beside the ray whose edge tests underflow to zero: the reference
    counts them as hit, at a distance that overflows.  All are in one leaf, so
    that a pass of the leaf phase finds many of them for one ray."""
    s = S.Scene("slivers")
    sliver = [(0, 0, 1e-6), (1e3, 0, 1e-6), (5e2, 1e-25, 1e-6)]
    v = sliver * 40 + [(0, -5, 0), (1e3, -5, 2e-6), (0, -4, 0)]
    s.add(S.MAT_DIFFUSE, np.array(v, np.float32), np.arange(len(v)).reshape(-1, 3))
    r = np.tile(np.array([-1, 0, 0, 2e-15, 0, 1.4e-45], np.float32), (100, 1))
    h = same_hits(pair, s, r)
    assert np.isinf(h["t"][h["tri"] != 0xFFFFFFFF]).all()


def test_long_directions_are_as_fast_as_unit_ones(pair):  # noqa: F811
    """2^20 rays of length 1 and 1e7 through the same mesh: the second batch may
    not take more than twice the first's time (left to the one-lane fallback it
    took sixteen times)."""
    import torch

    ctx, _ = pair
    s = S.icosphere_kd(6, seed=1)
    sid = ctx.upload(s)
    unit = torch.tensor(S.kd_rays(s, 1 << 20, seed=3), device="cuda")
    hits = torch.empty((len(unit), 4), dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    times = []
    for scale in (1.0, 1e7):
        rays = unit.clone()
        rays[:, 3:] *= scale
        torch.cuda.synchronize()
        best = np.inf
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            ctx.trace_closest_device(sid, rays.data_ptr(), len(rays), hits.data_ptr(), stream.cuda_stream)
            b.record(stream)
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    ctx.release(sid)
    assert times[1] < 2 * times[0], times
