"""The framework's work as its users call it, for timing and for comparing
outputs: closest-hit batches and render calls over the range of sizes,
options and scenes that the configurations, the tests and bench.py use.

A case is a dict of plain values.  Its "kind" names the entry point:

  rays        Context.trace_closest_device: rays and hits in device memory
  rays_host   Context.trace_closest: host arrays in, host arrays out
  film        Context.render_device: samples added to a device film
  image       Context.render: the mean image on the host
  serve       Server.submit / wait / fetch: several requests at once
"""
import functools
import math

import numpy as np
import torch

from walkray_gb300 import scenes as S
from walkray_gb300.api import LOW_VARIANCE, Context, Server


def listed():
    return [
        # a picking or probing call: a thousand rays against a small mesh, where latency counts
        {"name": "rays_1k", "kind": "rays", "scene": "ico", "level": 4, "n": 1009, "filtered": False},
        # one bounce of an integrator that lives outside the library: surface rays with NoSelfCondition's
        # inside / contact ids on the mixed-material scene, an odd count
        {"name": "rays_bounce_200k", "kind": "rays", "scene": "mixed", "level": 5, "n": 200003, "filtered": True},
        # the closest-hit microbenchmark: 1,310,720 triangles, 2^24 incoherent rays
        {"name": "rays_16m", "kind": "rays", "scene": "ico", "level": 8, "n": 1 << 24, "filtered": False},
        # a host program's batch: rays from host memory, hits back to it
        {"name": "rays_host_1m", "kind": "rays_host", "scene": "ico", "level": 5, "n": 1100003, "filtered": False},
        # an interactive preview frame: one sample per pixel, the image to the host
        {"name": "preview_cornell", "kind": "image", "scene": "cornell", "width": 160, "height": 120, "spp": 1,
         "depth": 8, "mode": "wavefront", "low_variance": False, "nee": False},
        # the plain Cornell box configuration: 256^2, 64 spp, depth 8
        {"name": "film_cornell", "kind": "film", "scene": "cornell", "width": 256, "height": 256, "spp": 64,
         "depth": 8, "mode": "wavefront", "low_variance": False, "nee": False},
        # the headline scene at its own resolution and depth; 32 of its 256 samples per pixel
        {"name": "film_mixed", "kind": "film", "scene": "mixed", "level": 5, "width": 1024, "height": 1024, "spp": 32,
         "depth": 16, "mode": "wavefront", "low_variance": False, "nee": False},
        # the same scene with the low-variance estimators (light connections through the shadow stage), a ragged size
        {"name": "image_mixed_low_variance", "kind": "image", "scene": "mixed", "level": 5, "width": 641, "height": 479,
         "spp": 16, "depth": 16, "mode": "wavefront", "low_variance": True, "nee": False},
        # participating media: the 128^3 density grid and a homogeneous sphere, depth 24
        {"name": "film_media", "kind": "film", "scene": "media", "width": 512, "height": 512, "spp": 16, "depth": 24,
         "mode": "wavefront", "low_variance": False, "nee": False},
        # the plain form of the renderer, a ragged size
        {"name": "megakernel_mixed", "kind": "image", "scene": "mixed", "level": 5, "width": 333, "height": 251,
         "spp": 8, "depth": 16, "mode": "megakernel", "low_variance": False, "nee": False},
        # bidirectional path tracing as bench.py runs it: Cornell box, 256^2, depth 8, 16 spp
        {"name": "bidirectional_cornell", "kind": "image", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "mode": "bidirectional", "low_variance": False, "nee": False},
        # the serving loop: requests of three scenes and several sizes in flight together
        {"name": "serve_six", "kind": "serve", "requests": 6, "largest": 512, "spp": 16, "level": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "rays", "rays", "rays_host", "film", "film", "film", "image", "image", "serve"])
    if kind in ("rays", "rays_host"):
        mixed = rng.random() < 0.4
        return {"kind": kind, "scene": "mixed" if mixed else "ico",
                "level": rng.randint(2, 5) if mixed else rng.randint(2, 8),
                "n": _log(rng, 500, 1 << (22 if kind == "rays" else 21)) | rng.randint(0, 1),
                "filtered": mixed and rng.random() < 0.7}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(2, 8), "largest": _log(rng, 96, 600), "spp": rng.randint(4, 24),
                "level": rng.randint(3, 5)}
    mode = rng.choice(["wavefront"] * 5 + ["megakernel", "bidirectional", "photon_map"])
    scene = rng.choice(["cornell", "mixed", "mixed", "media"])
    if mode in ("bidirectional", "photon_map"):
        scene = "cornell"
    c = {"kind": kind, "scene": scene, "width": _log(rng, 40, 1024), "height": _log(rng, 40, 1024),
         "depth": {"cornell": 8, "mixed": 16, "media": 24}[scene], "mode": mode, "low_variance": False, "nee": False}
    if scene == "mixed":
        c["level"] = rng.randint(3, 5)
    most = {"wavefront": 1 << (22 if scene == "media" else 24), "megakernel": 1 << 21}.get(mode, 1 << 20)
    c["spp"] = _log(rng, 1, max(1, min(64, most // (c["width"] * c["height"]))))
    if mode in ("wavefront", "megakernel"):
        c["low_variance"] = rng.random() < 0.3
        c["nee"] = not c["low_variance"] and rng.random() < 0.15
    return c


# ---------------------------------------------------------------------------
# scenes: the geometry is made once per process, as a program loads its files
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _mesh(level):
    return S.icosphere_kd(level, seed=1)


@functools.lru_cache(maxsize=None)
def _mixed(level):
    return S.mixed_spheres(64, 64, seed=7, level=level)


@functools.lru_cache(maxsize=None)
def _media():
    return S.cornell_media(64, 64)


def _scene(name, level=None, width=64, height=64):
    base = {"ico": lambda: _mesh(level), "mixed": lambda: _mixed(level), "cornell": lambda: S.cornell(64, 64),
            "media": _media}[name]()
    s = S.Scene(base.name)
    s.objects, s.grids, c = base.objects, base.grids, base.camera
    scale = height / c.height
    s.camera = S.Camera(c.position, c.focus, c.up, width, height, c.image_plane_dist * scale, c.lens_radius,
                        c.focal_dist)
    return s


@functools.lru_cache(maxsize=None)
def _program():
    # one context per program and one stream for its calls: calls of a context share its scratch memory, so a
    # program that put them on several streams would have to order them itself
    return Context(device=0), torch.cuda.Stream()


class _State:
    """What a program holds between calls; its scenes go with it."""

    def __init__(self):
        self.ctx, self.sids, self.server = None, [], None

    def __del__(self):
        try:
            if self.server is not None:
                self.server.stop()
                self.ctx.close()
            else:
                for sid in self.sids:
                    self.ctx.release(sid)
        except Exception:
            pass


def _uniform_rays(scene, n, gen):
    """bench.py's closest-hit rays: origins uniform in a box twice the mesh bounds, directions uniform."""
    v = np.concatenate([o.verts for o in scene.objects])
    lo, hi = v.min(0).astype(np.float64), v.max(0).astype(np.float64)
    c, h = torch.tensor((lo + hi) / 2, device="cuda"), torch.tensor((hi - lo) / 2, device="cuda")
    o = c + (torch.rand((n, 3), generator=gen, device="cuda") * 2 - 1) * (2 * h)
    d = torch.randn((n, 3), generator=gen, device="cuda")
    d = d / d.norm(dim=1, keepdim=True)
    return torch.cat([o.float(), d], 1).contiguous()


def _bounce_rays(scene, n, gen):
    """Rays as they leave surfaces: a random point of a random triangle, a direction of the cosine hemisphere
    above it (half of a refractive object's: below it, inside the object); inside and contact ids."""
    tri, vert = _triangles(scene)
    p = torch.tensor(vert, device="cuda", dtype=torch.float64)[torch.tensor(tri.astype(np.int64), device="cuda")]
    obj = torch.tensor(scene.tri_object_ids(), device="cuda", dtype=torch.int64)
    clear = torch.tensor([o.type == S.MAT_REFRACTIVE for o in scene.objects], device="cuda")
    k = torch.randint(0, len(p), (n,), generator=gen, device="cuda")
    a, b = torch.rand((2, n, 1), generator=gen, device="cuda", dtype=torch.float64)
    r = a.sqrt()
    v0, v1, v2 = p[k, 0], p[k, 1], p[k, 2]
    o = v0 * (1 - r) + v1 * (r * (1 - b)) + v2 * (r * b)
    nrm = torch.linalg.cross(v1 - v0, v2 - v0)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    d = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    d = nrm * 1.001 + d / d.norm(dim=1, keepdim=True)
    d = d / d.norm(dim=1, keepdim=True)
    contact = obj[k]
    inward = clear[contact] & (torch.rand((n,), generator=gen, device="cuda") < 0.5)
    d = torch.where(inward[:, None], d - 2 * (d * nrm).sum(1, keepdim=True) * nrm, d)
    inside = torch.where(inward, contact, torch.full_like(contact, -1))
    return torch.cat([o, d], 1).float().contiguous(), inside.int().contiguous(), contact.int().contiguous()


def _triangles(scene):
    return scene.global_triangles(), np.concatenate([o.verts for o in scene.objects])


def _inputs(case, scene, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["filtered"]:
        return _bounce_rays(scene, case["n"], gen)
    return _uniform_rays(scene, case["n"], gen), None, None


def prepare(case, seed):
    s = _State()
    s.case, s.seed = case, seed
    if case["kind"] == "serve":
        s.ctx = Context(device=0)
        g = np.random.default_rng(seed)
        kinds = ["cornell", "mixed", "media"]
        s.sids = [s.ctx.upload(_scene(k, case["level"])) for k in kinds]
        s.server = Server(s.ctx, film_bytes=1 << 28)
        s.requests = []
        for k in range(case["requests"]):
            side = max(16, case["largest"] >> (k % 3))  # every size for every seed: the same work
            spp = max(1, case["spp"] // (1 + k % 2))
            s.requests.append((s.sids[k % 3], side, side - side // 4, spp, (8, 16, 24)[k % 3], int(g.integers(1 << 30))))
        return s
    s.ctx, s.stream = _program()
    scene = _scene(case["scene"], case.get("level"), case.get("width", 64), case.get("height", 64))
    s.sids = [s.ctx.upload(scene)]
    if case["kind"] in ("rays", "rays_host"):
        s.rays, s.inside, s.contact = _inputs(case, scene, seed)
        if case["kind"] == "rays":
            s.hits = torch.empty((case["n"], 4), dtype=torch.int32, device="cuda")
        else:
            s.rays = s.rays.cpu().numpy()
            if case["filtered"]:
                s.inside, s.contact = s.inside.cpu().numpy(), s.contact.cpu().numpy()
    elif case["kind"] == "film":
        s.film = torch.empty((case["height"], case["width"], 3), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return s


def _render_options(s):
    c = s.case
    return dict(spp=c["spp"], max_path_len=c["depth"], seed=s.seed, mode=c["mode"], nee=c["nee"],
                flags=LOW_VARIANCE if c["low_variance"] else 0)


def run(s):
    c, kind = s.case, s.case["kind"]
    if kind == "rays":
        s.ctx.trace_closest_device(s.sids[0], s.rays.data_ptr(), c["n"], s.hits.data_ptr(), s.stream.cuda_stream,
                                   s.inside.data_ptr() if c["filtered"] else 0,
                                   s.contact.data_ptr() if c["filtered"] else 0)
        h = s.hits
        return {"tri": h[:, 0], "t": h.view(torch.float32)[:, 1], "u": h.view(torch.float32)[:, 2:]}
    if kind == "rays_host":
        h = s.ctx.trace_closest(s.sids[0], s.rays, s.inside, s.contact)
        h = h.view(np.uint32).reshape(-1, 4)
        f = h.view(np.float32)
        return {"tri": h[:, 0].astype(np.int64), "t": f[:, 1], "u": f[:, 2:]}
    if kind == "film":
        with torch.cuda.stream(s.stream):
            s.film.zero_()
            s.ctx.render_device(s.sids[0], d_sum=s.film.data_ptr(), stream=s.stream.cuda_stream, **_render_options(s))
        return s.film
    if kind == "image":
        return s.ctx.render(s.sids[0], **_render_options(s))
    ids = [s.server.submit(sid, w, h, spp, depth, seed=seed) for sid, w, h, spp, depth, seed in s.requests]
    s.server.wait(ids)
    return [s.server.fetch(i) for i in ids]


def _triangle_count(name, level):
    return {"ico": lambda: 20 * 4 ** level, "mixed": lambda: 25 * 20 * 4 ** level + 6, "cornell": lambda: 36,
            "media": lambda: 36 + 12 + 1280}[name]()


def _render_work(name, level, width, height, spp):
    # ray segments of a path and floating-point operations of one: a walk down the tree, a few triangles and
    # the bounce's shading (and the tracking steps through the density grid)
    segments = {"cornell": 3.0, "mixed": 3.0, "media": 6.0}[name]
    per = 20 * math.log2(_triangle_count(name, level)) + 300 + (400 if name == "media" else 0)
    grid = 4 * 128 ** 3 if name == "media" else 0
    return {"bytes": 12.0 * width * height + 36 * _triangle_count(name, level) + grid,
            "flops": width * height * spp * segments * per}


def work(case):
    if case["kind"] in ("rays", "rays_host"):
        t = _triangle_count(case["scene"], case["level"])
        return {"bytes": case["n"] * (48.0 if case["filtered"] else 40.0) + 36.0 * t,
                "flops": case["n"] * (20 * math.log2(t) + 100.0)}
    if case["kind"] == "serve":
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["requests"]):
            side = max(16, case["largest"] >> (k % 3))
            w = _render_work(("cornell", "mixed", "media")[k % 3], case["level"], side, side - side // 4,
                             max(1, case["spp"] // (1 + k % 2)))
            total = {m: total[m] + w[m] for m in total}
        return total
    return _render_work(case["scene"], case.get("level"), case["width"], case["height"], case["spp"])


def exact(case, seed):
    """Closest hits by testing every triangle in 64 bits (rays whose count times the triangles' stays moderate)."""
    if case["kind"] not in ("rays", "rays_host"):
        return None
    if case["n"] * _triangle_count(case["scene"], case["level"]) > 1.1e11:
        return None
    scene = _scene(case["scene"], case["level"])
    rays, inside, contact = _inputs(case, scene, seed)
    tri, vert = _triangles(scene)
    p = torch.tensor(vert, device="cuda", dtype=torch.float64)[torch.tensor(tri.astype(np.int64), device="cuda")]
    v = [p[:, k] for k in range(3)]
    cross = torch.linalg.cross
    # the signed volumes d . ((v1 - v0) x (v0 - o)) of the three edges as products of 6-vectors
    edge = [v[(k + 1) % 3] - v[k] for k in range(3)]
    plane = [torch.cat([cross(edge[k], v[k]), edge[k]], 1).T.contiguous() for k in range(3)]
    nrm = cross(edge[0], v[2] - v[0])
    off = (nrm * v[0]).sum(1)
    obj = torch.tensor(scene.tri_object_ids(), device="cuda", dtype=torch.int32)
    t_all = torch.full((case["n"],), -1.0, device="cuda", dtype=torch.float64)
    u_all = torch.zeros((case["n"], 2), device="cuda", dtype=torch.float64)
    step = max(1, (1 << 26) // len(p))
    for a in range(0, case["n"], step):
        o, d = rays[a:a + step, :3].double(), rays[a:a + step, 3:].double()
        od = torch.cat([d, -cross(o, d)], 1)
        ge = le = None
        for k in range(3):
            s = od @ plane[k]
            ge, le = (s >= 0, s <= 0) if ge is None else (ge & (s >= 0), le & (s <= 0))
        dn = d @ nrm.T
        t = (off[None, :] - o @ nrm.T) / dn
        ok = (ge | le) & (dn != 0) & (t >= 0)
        if case["filtered"]:
            i, c = inside[a:a + step, None], contact[a:a + step, None]
            hit = obj[None, :]
            legal = torch.where(i == c, ~((dn <= 0) & (c == hit)), ~((dn >= 0) & (i != hit)))
            ok &= legal
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, k = t.min(1)
        hit = torch.isfinite(best)
        e1, e2 = v[1][k] - v[0][k], v[2][k] - v[0][k]
        x = o + d * torch.where(hit, best, torch.zeros_like(best))[:, None] - v[0][k]
        n = cross(e1, e2)
        nn = (n * n).sum(1)
        u = torch.stack([(cross(x, e2) * n).sum(1) / nn, (cross(e1, x) * n).sum(1) / nn], 1)
        t_all[a:a + step] = torch.where(hit, best, torch.full_like(best, -1.0))
        u_all[a:a + step] = torch.where(hit[:, None], u, torch.zeros_like(u))
    return {"tri": None, "t": t_all, "u": u_all}
