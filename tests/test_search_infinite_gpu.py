"""Scenes with vertices that are not finite: the search's results are those of
the walk that visits every box the reference visits, bit for bit, with one such
vertex and with some in many leaves; one of them does not slow the other
triangles' rays down."""
import numpy as np
import pytest

from test_search_gpu import directions, pair, rays_of, same_hits, soup  # noqa: F401  (pair: a fixture)
from walkray_gb300 import scenes as S
from walkray_gb300.api import LOW_VARIANCE

pytestmark = pytest.mark.gpu
INF, NAN = np.inf, np.nan


def odd_scene(values, where, base):
    """The base mesh and, for each entry of `where`, a triangle with one of `values` in one coordinate."""
    rng = np.random.default_rng(4)
    s = S.Scene("odd")
    s.add(S.MAT_DIFFUSE, *base)
    for k, (vert, axis) in enumerate(where):
        v = rng.random((3, 3)).astype(np.float32)
        v[vert, axis] = values[k % len(values)]
        s.add(S.MAT_DIFFUSE, v, [(0, 1, 2)])
    return s


def finite_rays(s, n, kind):
    f = S.Scene("finite")
    f.objects = s.objects[:1]
    return rays_of(f, kind, n)


@pytest.mark.parametrize("kind", ["plain", "axis", "corners", "scaled", "odd"])
@pytest.mark.parametrize("values", [(INF,), (-INF,), (NAN,), (INF, -INF, NAN)], ids=["inf", "-inf", "nan", "all"])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 24, 25, 300, 2000])
def test_scenes_with_vertices_that_are_not_finite(pair, count, values, kind):  # noqa: F811
    rng = np.random.default_rng(count)
    where = [(int(rng.integers(3)), int(rng.integers(3))) for _ in range(count)]
    s = odd_scene(values, where, soup(300, rng, 0.3))
    same_hits(pair, s, finite_rays(s, 3000, kind))


@pytest.mark.parametrize("values", [(INF, INF, INF), (NAN, NAN, NAN), (INF, -INF, 0.0)])
def test_a_scene_of_such_triangles_alone(pair, values):  # noqa: F811
    s = S.Scene("odd")
    s.add(S.MAT_DIFFUSE, np.array([values, (1, 0, 0), (0, 1, 0)], np.float32), [(0, 1, 2)])
    rng = np.random.default_rng(2)
    same_hits(pair, s, np.concatenate([rng.random((3000, 3)), directions(3000, rng)], 1).astype(np.float32))


@pytest.mark.parametrize("options", [{}, {"nee": True}, {"flags": LOW_VARIANCE}], ids=["plain", "nee", "low_variance"])
@pytest.mark.parametrize("width,height", [(1, 1), (33, 1), (67, 61)])
def test_images_of_such_a_scene(ctx, width, height, options):
    """Wavefront against megakernel at one sample per pixel, so that each pixel is
    one path: the kernels' own rounding alone may differ (3e-5, as in the
    wavefront's stage tests)."""
    s = S.mixed_spheres(width, height, seed=7, level=2)
    rng = np.random.default_rng(1)
    for k in range(100):
        v = rng.random((3, 3)).astype(np.float32)
        v[k % 3, k // 3 % 3] = INF
        s.add(S.MAT_DIFFUSE, v, [(0, 1, 2)])
    sid = ctx.upload(s)
    a = ctx.render(sid, 1, 16, seed=5, mode="megakernel", **options)
    b = ctx.render(sid, 1, 16, seed=5, mode="wavefront", **options)
    ctx.release(sid)
    assert np.allclose(a, b, rtol=1e-4, atol=1e-5), np.abs(a - b).max()


def test_one_infinite_vertex_does_not_slow_the_search(pair):  # noqa: F811
    """2^19 rays through a mesh, without and with one more triangle that has an
    infinite vertex: at most four times the first's time (without a tree for the
    others it took some twenty times)."""
    import torch

    ctx, _ = pair
    stream = torch.cuda.Stream()
    mesh = S.icosphere_kd(6, seed=1)
    rays = torch.tensor(S.kd_rays(mesh, 1 << 19, seed=3), device="cuda")
    hits = torch.empty((len(rays), 4), dtype=torch.int32, device="cuda")
    times = []
    for odd in (False, True):
        if odd:
            mesh.add(S.MAT_DIFFUSE, np.array([(0, 0, 0), (1, 0, 0), (0, INF, 0)], np.float32), [(0, 1, 2)])
        sid = ctx.upload(mesh)
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
    assert times[1] < 4 * times[0], times
