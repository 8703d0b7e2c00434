"""The four-wide search (the default closest hit) against the walk that visits
every box the reference visits (WR_CTX_EXACT_TRAVERSAL): the same triangle ids
and the same t bit for bit, on the rays and scenes where the two could part --
box faces, edges and corners, flat boxes, leaves of many coincident triangles,
walks deeper than the stack, directions at the ends of the float range, values
that are not finite -- and at the sizes where the warps' queues and runs end."""
import numpy as np
import pytest

from walkray_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair():
    from walkray_gb300.api import Context

    with Context() as ctx, Context(exact_traversal=True) as ex:
        yield ctx, ex


def same_hits(pair, scene, rays, inside=None, contact=None):
    ctx, ex = pair
    a, b = ctx.upload(scene), ex.upload(scene)
    h, g = ctx.trace_closest(a, rays, inside, contact), ex.trace_closest(b, rays, inside, contact)
    ctx.release(a)
    ex.release(b)
    assert np.array_equal(h["tri"], g["tri"])
    for k in ("t", "b1", "b2"):
        assert np.array_equal(h[k].view(np.uint32), g[k].view(np.uint32)), k
    return h


def directions(n, rng):
    d = rng.standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def soup(n, rng, size=0.05):
    c = rng.random((n, 1, 3))
    v = (c + (rng.random((n, 3, 3)) - 0.5) * size).astype(np.float32)
    return v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def scene_of(name):
    rng = np.random.default_rng(3)
    s = S.Scene(name)
    if name == "cornell":
        return S.cornell()
    if name == "mixed":
        return S.mixed_spheres(level=3)
    if name == "empty":
        pass
    elif name == "one":
        s.add(S.MAT_DIFFUSE, [(0, 0, 0), (1, 0, 0), (0, 1, 0)], [(0, 1, 2)])
    elif name == "grid":  # axis-aligned quads that share edges: every box flat, every edge on a box edge
        x, y = np.meshgrid(np.arange(17), np.arange(17), indexing="ij")
        v = np.stack([x.ravel() / 16, y.ravel() / 16, np.full(17 * 17, 0.5)], 1)
        i = (np.arange(16)[:, None] * 17 + np.arange(16)[None, :]).ravel()
        s.add(S.MAT_DIFFUSE, v, np.concatenate([np.stack([i, i + 17, i + 18], 1), np.stack([i, i + 18, i + 1], 1)]))
    elif name == "coincident":  # leaves of 40 triangles: the same positions again and again
        v, f = soup(6, rng, 0.8)
        s.add(S.MAT_DIFFUSE, v, np.concatenate([f] * 40))
    elif name == "overlap":  # every box covers most of the scene: deep walks with many waiting children
        v, f = soup(4000, rng, 1.8)
        s.add(S.MAT_DIFFUSE, v, f)
    elif name == "soup":
        v, f = soup(5000, rng)
        s.add(S.MAT_DIFFUSE, v, f)
    elif name == "far":  # coordinates beyond the search's own range
        v, f = soup(500, rng, 0.5)
        s.add(S.MAT_DIFFUSE, v * np.float32(4e9), f)
    return s


def rays_of(scene, kind, n):
    rng = np.random.default_rng(11)
    v = np.concatenate([o.verts for o in scene.objects]) if scene.objects else np.zeros((1, 3), np.float32)
    lo, hi = v.min(0).astype(np.float64), v.max(0).astype(np.float64)
    o = lo - 0.3 * (hi - lo + 1e-3) + rng.random((n, 3)) * 1.6 * (hi - lo + 1e-3)
    d = directions(n, rng)
    if kind == "axis":  # zero and near-zero components, both signs of zero
        d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([0.0, -0.0, 1e-30, -1e-25, 1e-12], n)
        d[: n // 4] = np.eye(3)[rng.integers(0, 3, n // 4)] * rng.choice([-1, 1], (n // 4, 1))
        o[: n // 8] = v[rng.integers(0, len(v), n // 8)]
    elif kind == "corners":  # at vertices (box corners and edges among them), from vertices
        o[: n // 2] = v[rng.integers(0, len(v), n // 2)]
        d = v[rng.integers(0, len(v), n)] - o
        d[np.abs(d).sum(1) == 0] = (0.0, 0.0, 1.0)
    elif kind == "scaled":  # directions that are not of unit length
        d *= 10.0 ** rng.uniform(-9, 9, (n, 1))
    elif kind == "odd":  # zero, infinite and NaN values among ordinary rays
        k = n // 8
        d[:k] = 0.0
        d[k:2 * k, 0] = np.nan
        d[2 * k:3 * k, 1] = np.inf
        o[3 * k:4 * k, 2] = np.nan
        o[4 * k:5 * k] *= 1e12
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("kind", ["plain", "axis", "corners", "scaled", "odd"])
@pytest.mark.parametrize("scene", ["cornell", "mixed", "empty", "one", "grid", "coincident", "overlap", "soup", "far"])
def test_search_equals_the_reference_walk(pair, scene, kind):
    s = scene_of(scene)
    same_hits(pair, s, rays_of(s, kind, 20000))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 129, 4095, 34048, 34049, 1 << 18])
def test_search_at_the_ends_of_queues_and_runs(pair, n):
    s = scene_of("mixed")
    same_hits(pair, s, rays_of(s, "plain", n))


@pytest.mark.parametrize("scene", ["cornell", "mixed", "coincident"])
def test_search_with_noself_condition(pair, scene):
    s = scene_of(scene)
    n = 20000
    rng = np.random.default_rng(5)
    r = rays_of(s, "corners", n)
    inside = rng.integers(-1, len(s.objects), n).astype(np.int32)
    contact = rng.integers(-2, len(s.objects), n).astype(np.int32)
    contact[::3] = inside[::3]
    same_hits(pair, s, r, inside, contact)
