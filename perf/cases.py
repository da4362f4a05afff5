"""The work that users of the ray-query engine have it do, as cases that a timer can run.

Every case goes through the engine's public entry points (the ctypes binding of the C ABI)
with device buffers on torch's current stream, as a CUDA program holds them; the two whose
calls take host arrays by their nature (the reference render, the streamed host queries)
keep them on the host.  Meshes are seeded fBm terrains and displaced spheres, rays are
camera, bounce (cosine hemisphere), shadow and random rays, at the sizes of the benchmark,
of the tests and of the reference program's own scene, and ranges around them.

A case names what it does in "kind":
  pick      a few rays against a resident LBVH (mouse picking, probes): call latency
  lidar     new vertices, LBVH rebuild, one scan of rays (an animated mesh under a sensor)
  random    a batch of rays in no order against a resident LBVH
  step      new vertices, LBVH rebuild, camera + bounce + shadow queries (the benchmark's step)
  frame     new vertices, rebuild (LBVH, BVH or KDTREE), one rendered image with shadow rays
  reference the reference program's frame: median BVH over spheres, its camera and shading
  median    new vertices, median BVH rebuild, one scan of rays
  kd        bounce rays against a resident KD tree
  host      closest-hit and any-hit queries over host arrays (streamed), resident median BVH
  batch     many meshes: one batched LBVH rebuild and one many-structure query
"""
import functools
import importlib
import math

import numpy as np
import torch

rq = importlib.import_module("raytracer-data-structures_gb300.rq")

DEV = "cuda"
EYE, TARGET, FOV, LIGHT = (0.0, -0.6, 1.1), (0.0, 0.0, 0.0), 40.0, (1.5, -1.0, 3.0)
SPHERE_VIEW = dict(eye=(0.0, 0.0, 3.0), target=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), fov_deg=40.0,
                   light=(2.0, 3.0, 4.0), albedo=(0.8, 0.75, 0.7), ambient=0.1)
CLUSTER_VIEW = dict(eye=(0.0, -12.0, 5.0), target=(0.0, 0.0, 0.0), up=(0.0, 0.0, 1.0), fov_deg=50.0,
                    light=(6.0, -8.0, 10.0), albedo=(0.75, 0.7, 0.65), ambient=0.05, mirror=0.5, bounces=2)


# ------------------------------------------------------------------- cases

def listed():
    return [
        # The smallest call: a handful of probe rays against a 20k-triangle mesh.
        {"name": "pick", "kind": "pick", "n": 41, "rays": 1023},
        # The reference program's own workload (its bunny has 35,947 vertices, each a sphere, and a
        # floor sphere): median BVH and a 640x480 image, as main() does per run.
        {"name": "reference_frame", "kind": "reference", "spheres": 35948, "width": 640, "height": 480},
        # The small plain render: an 82k-triangle mesh that moves, 640x480 with one shadow ray.
        {"name": "frame_small", "kind": "frame", "acc": "LBVH", "mesh": "sphere", "n": 83, "width": 640, "height": 480,
         "spp": 1},
        # The same frame on the KD tree (the reference's second structure): build-bound.
        {"name": "kd_frame", "kind": "frame", "acc": "KDTREE", "mesh": "sphere", "n": 83, "width": 640, "height": 480,
         "spp": 1},
        # A 998,000-triangle terrain that changes under a 64-line scanner: the build with default settings.
        {"name": "lidar", "kind": "lidar", "nx": 1001, "ny": 500, "rays": 64 * 1801},
        # The benchmark's step: rebuild with its tuned settings, 8.3M camera rays, 8.3M bounce rays, 8.3M shadow rays.
        {"name": "terrain_step", "kind": "step", "nx": 1001, "ny": 500, "width": 1920, "height": 1080, "spp": 4},
        # Rays in no order (global illumination caches, physics): a million against 331k triangles.
        {"name": "random", "kind": "random", "n": 166, "rays": 1000003},
        # The median BVH on a changing mesh of odd size, few rays per triangle.
        {"name": "median_rebuild", "kind": "median", "nx": 701, "ny": 357, "rays": 65537},
        # KD walk: bounce rays in scan order on a resident tree.
        {"name": "kd_bounce", "kind": "kd", "nx": 501, "ny": 251, "rays": 2073600},
        # Rays and results in (pinned) host memory, two queries in one call, resident median BVH.
        {"name": "host_queries", "kind": "host", "nx": 501, "ny": 251, "rays": 6000000},
        # 64 meshes of 1k to 100k triangles rebuilt and queried at once (simulation environments).
        {"name": "many_scenes", "kind": "batch", "scenes": 64, "lo": 1000, "hi": 100000, "rays": 8000000},
        # The large render: 150 objects, 10.3M triangles, 3840x2160 at 4 samples, shadows and two mirror bounces.
        {"name": "frame_large", "kind": "frame", "acc": "LBVH", "mesh": "cluster", "objects": 150, "n": 77, "width": 3840,
         "height": 2160, "spp": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pick", "reference", "frame", "frame", "lidar", "step", "random", "median", "kd", "host", "batch"])
    c = {"kind": kind}
    if kind in ("pick", "random"):
        c["n"] = _log(rng, 9, 290)  # 1k to 1M triangles
        c["rays"] = _log(rng, 1, 4096) if kind == "pick" else _log(rng, 10000, 4000000)
    elif kind == "reference":
        c.update(spheres=_log(rng, 500, 150000), width=rng.randrange(63, 1281), height=rng.randrange(47, 721))
    elif kind == "frame":
        c.update(acc=rng.choice(["LBVH", "LBVH", "BVH", "KDTREE"]), width=rng.randrange(65, 1921),
                 height=rng.randrange(49, 1081), spp=rng.choice([1, 1, 2, 4]))
        if c["acc"] == "LBVH" and rng.random() < 0.5:
            c.update(mesh="cluster", objects=rng.randrange(2, 101), n=_log(rng, 12, 60))
        else:
            c.update(mesh="sphere", n=_log(rng, 9, 110 if c["acc"] == "KDTREE" else 290))
    elif kind == "batch":
        c.update(scenes=_log(rng, 2, 128), lo=_log(rng, 300, 3000), hi=_log(rng, 5000, 60000), rays=_log(rng, 20000, 6000000))
    else:  # terrains of 1k to 1M triangles
        nx = _log(rng, 24, 500 if kind in ("kd", "host") else 1000)
        c.update(nx=nx, ny=max(3, min(500, int(nx * rng.uniform(0.4, 1.1)))))
        if kind == "step":
            c.update(width=rng.randrange(161, 1601), height=rng.randrange(121, 901), spp=rng.choice([1, 2, 4]))
        elif kind in ("kd", "host"):
            c["rays"] = _log(rng, 20000, 2000000 if kind == "kd" else 6000000)
        else:
            c["rays"] = _log(rng, 1000, 400000)
    return c


# ------------------------------------------------------------------ meshes

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _noise(p, freq, g):
    """Value noise of points p (n, 3) in [-1, 1]: a random lattice, smoothstep blend."""
    m = int(2 * freq) + 3
    lattice = torch.rand((m, m, m), generator=g, device=DEV, dtype=torch.float64) * 2 - 1
    q = (p + 1.0) * freq
    i = q.floor().clamp(0, m - 2).long()
    w = q - i
    w = w * w * (3 - 2 * w)
    out = 0
    for k in range(8):
        d = [(k >> a) & 1 for a in range(3)]
        f = 1
        for a in range(3):
            f = f * (w[:, a] if d[a] else 1 - w[:, a])
        out = out + f * lattice[i[:, 0] + d[0], i[:, 1] + d[1], i[:, 2] + d[2]]
    return out


def _fbm(p, octaves, freq, g):
    return sum(0.5 ** o * _noise(p, freq * 2 ** o, g) for o in range(octaves)) / sum(0.5 ** o for o in range(octaves))


@functools.lru_cache(maxsize=8)
def _grid_tris(nx, ny):
    i = (torch.arange(ny - 1, device=DEV)[:, None] * nx + torch.arange(nx - 1, device=DEV)[None, :]).reshape(-1)
    a, b, c, d = i, i + 1, i + nx, i + nx + 1
    return torch.stack([torch.stack([a, b, d], 1), torch.stack([a, d, c], 1)], 1).reshape(-1, 3).to(torch.int32)


def _terrain(nx, ny, seed):
    """fBm heights over [-1, 1]^2: vertices (ny * nx, 3) float32 and 2 (nx - 1)(ny - 1) triangles."""
    g = _gen(seed)
    x = torch.linspace(-1, 1, nx, device=DEV, dtype=torch.float64)
    y = torch.linspace(-1, 1, ny, device=DEV, dtype=torch.float64)
    p = torch.stack([x[None, :].expand(ny, nx).reshape(-1), y[:, None].expand(ny, nx).reshape(-1),
                     torch.zeros(nx * ny, device=DEV, dtype=torch.float64)], 1)
    z = 0.3 * _fbm(p, 5, 2.0, g)
    return torch.stack([p[:, 0], p[:, 1], z], 1).float().contiguous(), _grid_tris(nx, ny)


@functools.lru_cache(maxsize=8)
def _cube_sphere(n):
    """Unit sphere of six n x n faces: 12 n^2 triangles."""
    s = torch.linspace(-1, 1, n + 1, device=DEV, dtype=torch.float64)
    u, v = s[None, :].expand(n + 1, n + 1).reshape(-1), s[:, None].expand(n + 1, n + 1).reshape(-1)
    w = torch.ones_like(u)
    faces = [(u, v, w), (v, u, -w), (w, u, v), (-w, v, u), (v, w, u), (u, -w, v)]
    p = torch.cat([torch.stack(f, 1) for f in faces])
    t = _grid_tris(n + 1, n + 1)
    tris = torch.cat([t + k * (n + 1) ** 2 for k in range(6)]).to(torch.int32)
    return p / p.norm(dim=1, keepdim=True), tris.contiguous()


def _sphere(n, seed, radius=0.5):
    p, t = _cube_sphere(n)
    r = 1 + 0.15 * _fbm(p, 3, 2.0, _gen(seed))
    return (p * (radius * r)[:, None]).float().contiguous(), t


def _cluster(objects, n, seed):
    """Displaced spheres scattered over [-4, 4]^3, their resolutions around n."""
    r = np.random.default_rng(seed)
    vs, ts, off = [], [], 0
    for k in range(objects):
        v, t = _sphere(max(3, int(n * r.uniform(0.5, 1.4))), seed + 31 * k, r.uniform(0.05, 0.3))
        c = torch.tensor(r.uniform(-4, 4, 3), device=DEV, dtype=torch.float32)
        vs.append(v + c)
        ts.append(t + off)
        off += len(v)
    return torch.cat(vs), torch.cat(ts).to(torch.int32)


def _mesh(case, seed):
    if case.get("mesh") == "cluster":
        return _cluster(case["objects"], case["n"], seed)
    return _sphere(case["n"], seed) if "n" in case else _terrain(case["nx"], case["ny"], seed)


def _bunny_like(n, seed):
    """Sphere centres where the reference's scene has them: a displaced ball of small spheres and the floor sphere."""
    g = _gen(seed)
    p = torch.randn((n - 1, 3), generator=g, device=DEV, dtype=torch.float64)
    p = p / p.norm(dim=1, keepdim=True)
    c = p * (3.6 * (1 + 0.2 * _fbm(p, 3, 2.0, g)))[:, None] + torch.tensor([-2.0, 5.0, -58.0], device=DEV, dtype=torch.float64)
    s = torch.cat([c, torch.full((n - 1, 1), 0.05, device=DEV, dtype=torch.float64)], 1)
    floor = torch.tensor([[0.9359, -105.471, -43.236, 100.0]], device=DEV, dtype=torch.float64)
    return torch.cat([s, floor]).float().contiguous()


# -------------------------------------------------------------------- rays

def _pack(o, d, tmax=math.inf):
    """rq_ray_t records as an (n, 8) float32 tensor."""
    r = torch.zeros((len(d), 8), device=DEV, dtype=torch.float32)
    r[:, 0:3], r[:, 4:7], r[:, 7] = o, d, tmax
    return r


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _camera(width, height, spp, eye, target, fov, g):
    eye = np.asarray(eye, np.float64)
    w = np.asarray(target, np.float64) - eye
    w /= np.linalg.norm(w)
    u = np.cross(w, np.array([0.0, 0.0, 1.0]))
    u /= np.linalg.norm(u)
    v = np.cross(u, w)
    th = math.tan(math.radians(fov) / 2)
    n = width * height * spp
    pix = torch.arange(n, device=DEV) // spp
    j = torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64)
    sx = (2 * (pix % width + j[:, 0]) / width - 1) * th * (width / height)
    sy = (1 - 2 * (pix // width + j[:, 1]) / height) * th
    d = sx[:, None] * torch.tensor(u, device=DEV) + sy[:, None] * torch.tensor(v, device=DEV) + torch.tensor(w, device=DEV)
    return _pack(torch.tensor(eye, device=DEV), _unit(d))


def _surface(case, verts, n, g, window):
    """n points of the terrain in scan order over a window of it, and their normals."""
    nx, ny = case["nx"], case["ny"]
    rows = max(1, int(math.sqrt(n * 9 / 16)))
    cols = -(-n // rows)
    k = torch.arange(n, device=DEV)
    j = torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64)
    x = window[0] + (k % cols + j[:, 0]) / cols * (window[1] - window[0])
    y = window[3] - (k // cols + j[:, 1]) / rows * (window[3] - window[2])
    fx, fy = ((x + 1) / 2 * (nx - 1)).clamp(0, nx - 1.001), ((y + 1) / 2 * (ny - 1)).clamp(0, ny - 1.001)
    cx, cy = fx.long().clamp(max=nx - 2), fy.long().clamp(max=ny - 2)
    a, b = fx - cx, fy - cy
    tri = _grid_tris(nx, ny)[2 * (cy * (nx - 1) + cx) + (b > a).long()].long()
    p0, p1, p2 = (verts[tri[:, m]].double() for m in range(3))
    nrm = _unit(torch.linalg.cross(p1 - p0, p2 - p0))
    up = torch.minimum(a, b)[:, None]
    # lower triangle (v00, v10, v11): p0 + (a - b) (p1 - p0) + b (p2 - p0) ...; upper one alike
    lo = (b <= a)[:, None]
    p = torch.where(lo, p0 + (a[:, None] - up) * (p1 - p0) + up * (p2 - p0),
                    p0 + (b[:, None] - up) * (p2 - p0) + up * (p1 - p0))
    return p + 1e-4 * nrm, nrm


def _bounce(case, verts, n, g, window=(-0.8, 0.8, -0.6, 0.6)):
    """Cosine-weighted hemisphere rays from surface points in scan order."""
    p, nrm = _surface(case, verts, n, g, window)
    r = torch.rand((n, 2), generator=g, device=DEV, dtype=torch.float64)
    phi, sr = 2 * math.pi * r[:, 0], r[:, 1].sqrt()
    ax = torch.where((nrm[:, 0:1].abs() > 0.9), torch.tensor([[0.0, 1.0, 0.0]], device=DEV, dtype=torch.float64),
                     torch.tensor([[1.0, 0.0, 0.0]], device=DEV, dtype=torch.float64))
    t1 = _unit(torch.linalg.cross(nrm, ax))
    t2 = torch.linalg.cross(nrm, t1)
    d = (phi.cos() * sr)[:, None] * t1 + (phi.sin() * sr)[:, None] * t2 + (1 - r[:, 1]).sqrt()[:, None] * nrm
    return _pack(p, d)


def _shadow(case, verts, n, g, window=(-0.8, 0.8, -0.6, 0.6)):
    p, _ = _surface(case, verts, n, g, window)
    d = torch.tensor([LIGHT], device=DEV, dtype=torch.float64) - p
    dist = d.norm(dim=1)
    return _pack(p, d / dist[:, None], dist.float())


def _random(lo, hi, n, g):
    """Origins on a bounding sphere toward points in the box."""
    lo, hi = lo.double(), hi.double()
    s = _unit(torch.randn((n, 3), generator=g, device=DEV, dtype=torch.float64))
    o = (lo + hi) / 2 + s * (hi - lo).norm() / 2 * 1.05
    t = lo + torch.rand((n, 3), generator=g, device=DEV, dtype=torch.float64) * (hi - lo)
    return _pack(o, _unit(t - o))


def _scan(n, g):
    """A scanner above the terrain: lines of rays at growing angles from one origin."""
    k = torch.arange(n, device=DEV, dtype=torch.float64)
    az = 2 * math.pi * (k % 1801) / 1801 + 1e-3
    el = math.radians(12) + math.radians(68) * (k // 1801 + torch.rand(n, generator=g, device=DEV, dtype=torch.float64)) / (n // 1801 + 1)
    d = torch.stack([el.cos() * az.cos(), el.cos() * az.sin(), -el.sin()], 1)
    return _pack(torch.tensor([0.05, -0.07, 0.6], device=DEV, dtype=torch.float64), d)


def _batch(case, seed):
    """The meshes of a batch case, their rays back to back and the ray offsets."""
    r = np.random.default_rng(seed)
    share = r.uniform(0.2, 1.0, case["scenes"])
    cuts = np.round(np.cumsum(share) / share.sum() * case["rays"]).astype(np.int64)
    counts = np.diff(cuts, prepend=0)
    meshes, rays = [], []
    for k in range(case["scenes"]):
        tris = math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))
        if r.random() < 0.5:
            m = _sphere(max(2, int(math.sqrt(tris / 12))), seed + 7 * k)
        else:
            side = max(3, int(math.sqrt(tris / 2)) + 1)
            m = _terrain(side, side, seed + 7 * k)
        meshes.append(m)
        rays.append(_random(m[0].min(0).values, m[0].max(0).values, int(counts[k]), _gen(seed + 7 * k + 3)))
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    return meshes, torch.cat(rays), offs


def _inputs(case, seed):
    """What a case's program holds before the call: (vertices, triangles, {query: rays})."""
    seed = int(seed)
    if case["kind"] in ("reference", "batch"):
        raise ValueError("no mesh inputs")
    verts, tris = _mesh(case, seed)
    g = _gen(seed + 1000003)
    kind = case["kind"]
    if kind in ("pick", "random"):
        return verts, tris, {"hits": _random(verts.min(0).values, verts.max(0).values, case["rays"], g)}
    if kind in ("lidar", "median"):
        return verts, tris, {"hits": _scan(case["rays"], g)}
    if kind == "kd":
        return verts, tris, {"hits": _bounce(case, verts, case["rays"], g, (-1, 1, -1, 1))}
    if kind == "host":
        return verts, tris, {"hits": _bounce(case, verts, case["rays"], g), "shadow": _shadow(case, verts, case["rays"], g)}
    if kind == "step":
        n = case["width"] * case["height"] * case["spp"]
        return verts, tris, {"camera": _camera(case["width"], case["height"], case["spp"], EYE, TARGET, FOV, g),
                             "bounce": _bounce(case, verts, n, g), "shadow": _shadow(case, verts, n, g)}
    return verts, tris, {}


# ------------------------------------------------------------ prepare, run

class _State:
    """A program's handles and buffers; the engine's are closed with it."""

    def __init__(self, case, **settings):
        self.case, self.scenes, self.accels = case, [], []
        self.eng = rq.Engine(0, rq.default_settings(**settings))
        self.eng.set_stream(torch.cuda.current_stream().cuda_stream)

    def mesh(self, verts, tris):
        self.scenes.append(self.eng.scene_triangles(verts, tris))
        return self.scenes[-1]

    def __del__(self):
        for h in self.accels + self.scenes + [self.eng]:
            h.close()


def _hits(n):
    return torch.empty((n, 4), device=DEV, dtype=torch.float32)


def _fields(h):
    """rq_hit_t records as their fields."""
    return {"t": h[:, 0], "prim": h.view(torch.int32)[:, 1], "u": h[:, 2], "v": h[:, 3]}


def _bits(n):
    return torch.empty((n + 31) // 32, device=DEV, dtype=torch.int32)


def _view(case, seed):
    kw = CLUSTER_VIEW if case["mesh"] == "cluster" else SPHERE_VIEW
    return rq.make_view(seed=int(seed) + 11, **kw)


def _host_rays(r):
    h = torch.empty((len(r), 8), dtype=torch.float32, pin_memory=True)
    h.copy_(r)
    return h.numpy().view(rq.RAY_DTYPE).reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "reference":
        s = _State(case, width=case["width"], height=case["height"])
        sph = _bunny_like(case["spheres"], seed)
        s.scenes.append(s.eng.scene_spheres(sph))
        s.accels.append(s.eng.build(s.scenes[0], "BVH"))
        s.data = sph
        s.colors = np.tile(np.array([0.8, 0.7, 0.0], np.float32), (case["spheres"], 1))
        s.colors[-1] = 0.0
        return s
    if kind == "batch":
        s = _State(case)
        s.meshes, s.rays, s.offs = _batch(case, seed)
        s.accels = s.eng.build_batched([s.mesh(v, t) for v, t in s.meshes], "LBVH")
        s.hits = _hits(len(s.rays))
        return s
    verts, tris, rays = _inputs(case, seed)
    if kind == "frame":
        s = _State(case, width=case["width"], height=case["height"], aa_samples=case["spp"])
        s.view = _view(case, seed)
        s.pixels = torch.empty((case["height"], case["width"], 3), device=DEV, dtype=torch.uint8)
        s.rgb = torch.empty((case["height"], case["width"], 3), device=DEV, dtype=torch.float32)
    elif kind == "step":
        s = _State(case, morton=rq.MORTON_SCENE_CUBE, lbvh_quality=rq.LBVH_TREELETS)
        s.bounced = rq.default_settings(morton=rq.MORTON_SCENE_CUBE, lbvh_quality=rq.LBVH_TREELETS,
                                        ray_sort=rq.RAY_SORT_OCTANT)
        s.plain = s.eng.settings
    else:
        s = _State(case)
    acc = {"median": "BVH", "host": "BVH", "kd": "KDTREE", "frame": case.get("acc")}.get(kind, "LBVH")
    s.data = verts
    s.accels.append(s.eng.build(s.mesh(verts, tris), acc))
    if kind == "host":
        s.rays = {k: _host_rays(r) for k, r in rays.items()}
        n = case["rays"]
        s.hits = torch.empty((n, 4), dtype=torch.float32, pin_memory=True).numpy().view(rq.HIT_DTYPE).reshape(-1)
        s.bits = torch.empty((n + 31) // 32, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    else:
        s.rays = rays
        s.out = {k: _bits(len(r)) if k == "shadow" else _hits(len(r)) for k, r in rays.items()}
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "reference":
        s.scenes[0].update(s.data)
        s.accels[0].rebuild()
        pixels, rgb = s.eng.render_reference(s.accels[0], None, None, s.colors)
        return {"pixels": pixels, "rgb": rgb}
    if kind == "batch":
        for sc, (v, _) in zip(s.scenes, s.meshes):
            sc.update(v)
        s.eng.rebuild_batched(s.accels)
        s.eng.trace_batched(s.accels, s.rays, s.offs, out=s.hits)
        return _fields(s.hits)
    acc = s.accels[0]
    if kind == "host":
        s.eng.trace_queries(acc, [(s.rays["hits"], 0, s.hits, -1, -1), (s.rays["shadow"], 1, s.bits, -1, -1)])
        return {"t": s.hits["t"], "prim": s.hits["prim"].view(np.int32), "u": s.hits["u"], "v": s.hits["v"],
                "shadow": s.bits.view(np.int32)}
    if kind in ("pick", "random", "kd"):
        return _fields(s.eng.trace_closest(acc, s.rays["hits"], s.out["hits"]))
    s.scenes[0].update(s.data)
    acc.rebuild()
    if kind == "frame":
        s.eng.render(acc, s.view, s.pixels, s.rgb)
        return {"pixels": s.pixels, "rgb": s.rgb}
    if kind == "step":
        s.eng.trace_closest(acc, s.rays["camera"], s.out["camera"])
        s.eng.settings = s.bounced  # the tuned ray order of the incoherent query
        s.eng.trace_closest(acc, s.rays["bounce"], s.out["bounce"])
        s.eng.settings = s.plain
        s.eng.trace_any(acc, s.rays["shadow"], s.out["shadow"])
        return {"camera": _fields(s.out["camera"]), "bounce": _fields(s.out["bounce"]), "shadow": s.out["shadow"]}
    return _fields(s.eng.trace_closest(acc, s.rays["hits"], s.out["hits"]))


# -------------------------------------------------------------------- work

def _tris(case):
    if case.get("mesh") == "cluster":
        return int(case["objects"] * 12 * (case["n"] * 0.95) ** 2)
    return 12 * case["n"] ** 2 if "n" in case else 2 * (case["nx"] - 1) * (case["ny"] - 1)


def work(case):
    """Inputs read once, outputs written once: vertices (6 B a triangle of a grid) and indices, rays, hits or pixels.
    flops: one box test and a half a ray and tree level, two triangle tests a ray."""
    kind = case["kind"]
    if kind == "reference":
        n, q = case["spheres"], case["width"] * case["height"]
        return {"bytes": 16 * n + 12 * n + 15 * q, "flops": q * (math.log2(n) * 30 + 40) + 40 * n}
    if kind == "frame":
        n, q = _tris(case), case["width"] * case["height"]
        return {"bytes": 18 * n + 15 * q, "flops": 2 * q * case["spp"] * (math.log2(n) * 30 + 100) + 40 * n}
    if kind == "batch":
        n = int(case["scenes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]))
        return {"bytes": 18 * n + 48 * case["rays"], "flops": case["rays"] * 600 + 40 * n}
    n = _tris(case)
    if kind == "step":
        q = case["width"] * case["height"] * case["spp"]
        return {"bytes": 18 * n + q * (48 + 48 + 32.125), "flops": 3 * q * (math.log2(n) * 30 + 100) + 40 * n}
    q = case["rays"]
    return {"bytes": 18 * n + q * (48 + (32.125 if kind == "host" else 0)),
            "flops": (2 if kind == "host" else 1) * q * (math.log2(n) * 30 + 100)}


# ------------------------------------------------------------------- exact

def _closest64(v0, e1, e2, rays, block=128):
    """Closest hits in 64 bits: rays against boxes of `block` consecutive triangles, then the triangles of the boxes met."""
    n = len(v0)
    pad = -n % block
    if pad:
        z = torch.zeros((pad, 3), device=DEV, dtype=torch.float64)
        v0, e1, e2 = torch.cat([v0, v0[-1:].expand(pad, 3)]), torch.cat([e1, z]), torch.cat([e2, z])
    tri = [x.reshape(-1, block, 3) for x in (v0, e1, e2)]
    pts = torch.cat([tri[0], tri[0] + tri[1], tri[0] + tri[2]], 1)
    lo, hi = pts.min(1).values - 1e-6, pts.max(1).values + 1e-6
    m = len(rays)
    out = {k: torch.zeros(m, device=DEV, dtype=torch.float64) for k in ("t", "u", "v")}
    prim = torch.full((m,), -1, device=DEV, dtype=torch.int64)
    step = max(64, int(6e7 / len(lo)))
    for s in range(0, m, step):
        r = rays[s:s + step].double()
        o, d, t0, t1 = r[:, 0:3], r[:, 4:7], r[:, 3], r[:, 7]
        near, far = t0[:, None].clone(), t1[:, None].clone()
        for a in range(3):
            inv = 1 / d[:, a:a + 1]
            x, y = (lo[None, :, a] - o[:, a:a + 1]) * inv, (hi[None, :, a] - o[:, a:a + 1]) * inv
            near, far = torch.maximum(near, torch.minimum(x, y)), torch.minimum(far, torch.maximum(x, y))
        ri, bi = (near <= far).nonzero(as_tuple=True)
        best = t1.clone()
        bt = torch.full((len(r),), math.inf, device=DEV, dtype=torch.float64)
        bu, bv, bp = torch.zeros_like(bt), torch.zeros_like(bt), torch.full((len(r),), -1, device=DEV, dtype=torch.int64)
        for k in range(0, len(ri), 200000):
            i, b = ri[k:k + 200000], bi[k:k + 200000]
            p, f, g = (x[b] for x in tri)
            oo, dd = o[i][:, None, :], d[i][:, None, :].expand(-1, block, -1)
            pv = torch.linalg.cross(dd, g)
            det = (f * pv).sum(2)
            inv = 1 / det
            tv = oo - p
            u = (tv * pv).sum(2) * inv
            qv = torch.linalg.cross(tv, f)
            v = (dd * qv).sum(2) * inv
            t = (g * qv).sum(2) * inv
            ok = (det.abs() >= 1e-6) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > t0[i][:, None]) & (t < best[i][:, None])
            t = torch.where(ok, t, math.inf)
            tb, at = t.min(1)
            fin = torch.isfinite(tb)
            i, tb, at, row = i[fin], tb[fin], at[fin], fin.nonzero()[:, 0]
            old = bt.clone()
            bt.scatter_reduce_(0, i, tb, "amin")
            win = (tb == bt[i]) & (tb < old[i])
            w = i[win]
            bu[w], bv[w], bp[w] = u[row[win], at[win]], v[row[win], at[win]], (b[row[win]] * block + at[win])
        hit = torch.isfinite(bt) & (bp >= 0)
        out["t"][s:s + step] = torch.where(hit, bt, t1)
        out["u"][s:s + step], out["v"][s:s + step] = bu, bv
        prim[s:s + step] = torch.where(hit, bp, -1)
    return out, prim


def _tri64(verts, tris):
    p = [verts[tris[:, k].long()].double() for k in range(3)]
    # the engine's payload holds 32-bit edges
    return p[0], (p[1].float() - p[0].float()).double(), (p[2].float() - p[0].float()).double()


def _mix64(x):
    def shr(a, k):
        return (a >> k) & ((1 << (64 - k)) - 1)
    c = [v - (1 << 64) if v >= 1 << 63 else v for v in (0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB)]
    x = x + c[0]
    x = (x ^ shr(x, 30)) * c[1]
    x = (x ^ shr(x, 27)) * c[2]
    return x ^ shr(x, 31)


def _frame64(case, seed):
    """rq_render's image without mirror bounces, in 64 bits."""
    verts, tris, _ = _inputs(case, seed)
    kw = SPHERE_VIEW
    w, h, spp = case["width"], case["height"], case["spp"]
    f64 = lambda x: torch.tensor(x, device=DEV, dtype=torch.float64)  # noqa: E731
    n = w * h * spp
    r = torch.arange(n, device=DEV)
    pix = r // spp
    jit = [((_mix64((int(seed) + 11) ^ _mix64(r * 2 + k)) >> 40) & 0xFFFFFF).double() * 2.0 ** -24 for k in (0, 1)]
    eye, light = f64(kw["eye"]), f64(kw["light"])
    fwd = f64(kw["target"]) - eye
    fwd = fwd / fwd.norm()
    right = torch.linalg.cross(fwd, f64(kw["up"]))
    right = right / right.norm()
    up = torch.linalg.cross(right, fwd)
    th = math.tan(math.radians(kw["fov_deg"]) / 2)
    px = (2 * (pix % w + jit[0]) / w - 1) * th * (w / h)
    py = (1 - 2 * (pix // w + jit[1]) / h) * th
    d = _unit(fwd + px[:, None] * right + py[:, None] * up)
    inf = torch.full((n, 1), math.inf, device=DEV, dtype=torch.float64)
    zero = torch.zeros((n, 1), device=DEV, dtype=torch.float64)
    tri = _tri64(verts, tris)
    hit, prim = _closest64(*tri, torch.cat([eye.expand(n, 3), zero, d, inf], 1))
    live = prim >= 0
    q = prim[live]
    p = eye + d[live] * hit["t"][live][:, None]
    nrm = _unit(torch.linalg.cross(tri[1][q], tri[2][q]))
    nrm = torch.where((nrm * d[live]).sum(1, keepdim=True) > 0, -nrm, nrm)
    lv = light - p
    dist = lv.norm(dim=1, keepdim=True)
    ndl = (nrm * lv / dist).sum(1)
    _, blocked = _closest64(*tri, torch.cat([p + 1e-4 * nrm, zero[live], lv / dist, dist], 1))
    shade = kw["ambient"] + torch.where((blocked < 0) & (ndl > 0), ndl, 0.0)
    c = torch.ones((n, 3), device=DEV, dtype=torch.float64)
    c[live] = f64(kw["albedo"]) * shade[:, None]
    return {"pixels": None, "rgb": c.reshape(h, w, spp, 3).mean(2)}


def _reference64(case, seed):
    """The reference program's image in 64 bits (sum over its one sample a pixel)."""
    w, h = case["width"], case["height"]
    sph = _bunny_like(case["spheres"], seed).double()
    n = w * h
    bg = np.random.MT19937()
    bg._legacy_seeding(5489)
    raw = bg.random_raw(4 * n).astype(np.float64).reshape(-1, 2)
    jit = torch.tensor((raw[:, 0] + raw[:, 1] * 2.0 ** 32) / 2.0 ** 64, device=DEV).reshape(n, 2)
    pix = torch.arange(n, device=DEV)
    angle = math.tan(math.pi * 0.5 * 30 / 180)
    x = (2 * ((pix % w + jit[:, 0]) / w) - 1) * angle * (w / h)
    y = (1 - 2 * ((pix // w + jit[:, 1]) / h)) * angle
    d = _unit(torch.stack([x, y, -torch.ones_like(x)], 1))
    best, who = torch.full((n,), math.inf, device=DEV, dtype=torch.float64), torch.full((n,), -1, device=DEV)
    step = max(64, int(4e7 / len(sph)))
    l2, r2 = (sph[:, :3] ** 2).sum(1), sph[:, 3] ** 2
    for s in range(0, n, step):
        tca = d[s:s + step] @ sph[:, :3].T
        d2 = l2 - tca * tca
        thc = (r2 - d2).clamp(min=0).sqrt()
        t = torch.where(tca - thc < 0, tca + thc, tca - thc)
        t = torch.where((tca >= 0) & (d2 <= r2), t, math.inf)
        best[s:s + step], who[s:s + step] = t.min(1)
    live = torch.isfinite(best)
    c = torch.tensor([[0.6, 0.8, 1.0]], device=DEV, dtype=torch.float64).repeat(n, 1)
    p, dl, q = d[live] * best[live][:, None], d[live], who[live]
    nrm = _unit(p - sph[q, :3])
    nrm = torch.where((nrm * dl).sum(1, keepdim=True) > 0, -nrm, nrm)
    lv = _unit(torch.tensor([0.0, 3.0, 30.0], device=DEV, dtype=torch.float64) - p)
    amt = (lv * nrm).sum(1).clamp(min=0)
    refl = -lv + nrm * (2 * (lv * nrm).sum(1, keepdim=True))
    spec = (-(refl * dl).sum(1)).clamp(min=0) ** 25
    base = torch.tensor([0.815, 0.235, 0.031], device=DEV, dtype=torch.float64) * 0.8
    own = torch.where((q == len(sph) - 1)[:, None], 0.0, torch.tensor([0.8, 0.7, 0.0], device=DEV, dtype=torch.float64))
    c[live] = amt[:, None] * base / 2 + spec[:, None] * 0.5 + own
    return {"pixels": None, "rgb": c}


MOST_PAIRS = 8e9  # (ray, block of triangles) pairs that the 64-bit search takes on in its time


def exact(case, seed):
    kind = case["kind"]
    if kind == "reference":
        return _reference64(case, seed) if case["spheres"] * case["width"] * case["height"] < 1e11 else None
    if kind == "batch":
        n = case["scenes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        if case["rays"] * n / case["scenes"] / 128 > MOST_PAIRS:
            return None
        meshes, rays, offs = _batch(case, seed)
        parts = [_closest64(*_tri64(*m), rays[int(offs[k]):int(offs[k + 1])])[0] for k, m in enumerate(meshes)]
        out = {f: torch.cat([p[f] for p in parts]) for f in ("t", "u", "v")}
        return {"t": out["t"], "prim": None, "u": out["u"], "v": out["v"]}
    if kind == "frame":
        if case["mesh"] == "cluster" or 2 * case["width"] * case["height"] * case["spp"] * _tris(case) / 128 > MOST_PAIRS:
            return None
        return _frame64(case, seed)
    q = 2 * case["width"] * case["height"] * case["spp"] if kind == "step" else case["rays"]
    if q * _tris(case) / 128 > MOST_PAIRS:
        return None
    verts, tris, rays = _inputs(case, seed)
    tri = _tri64(verts, tris)
    found = {}
    for name, r in rays.items():
        if name == "shadow":
            found[name] = None
        else:
            h, _ = _closest64(*tri, r)
            found[name] = {"t": h["t"], "prim": None, "u": h["u"], "v": h["v"]}
    if kind == "host":
        return {**found["hits"], "shadow": None}
    return found if kind == "step" else found["hits"]
