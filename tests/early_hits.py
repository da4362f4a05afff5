"""Long triangles seen edge-on by rays whose Moller-Trumbore t lies well before
the triangle's box, each with a small triangle across the ray between the two:
which of them a walk answers depends on what it visits first."""
import numpy as np

import scenes

F = np.float32


def _cross(a, b):
    return np.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                     a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], 1)


def _dot(a, b):
    return (a[:, 0] * b[:, 0] + a[:, 1] * b[:, 1]) + a[:, 2] * b[:, 2]


def _mt(v0, v1, v2, o, d):
    """The engine's triangle test in float32: (accepted, t)."""
    e1, e2 = v1 - v0, v2 - v0
    p = _cross(d, e2)
    det = _dot(e1, p)
    with np.errstate(all="ignore"):
        inv = F(1) / det
        tv = o - v0
        u = _dot(tv, p) * inv
        q = _cross(tv, e1)
        v = _dot(d, q) * inv
        t = _dot(e2, q) * inv
        ok = (np.abs(det) >= F(1e-6)) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1)
    return ok, t


def scene_and_rays(n_pairs, seed):
    """(vertices, triangles, rays): n_pairs rays in doubt over their pairs and an ordinary sphere mesh around them."""
    rng = np.random.default_rng(seed)
    unit = lambda x: x / np.linalg.norm(x, axis=1, keepdims=True)  # noqa: E731
    long_t, small_t, org, dirs = [], [], [], []
    while sum(map(len, org)) < n_pairs:
        m = 400_000
        c = rng.uniform(-1, 1, (m, 3))
        v = [c + rng.normal(0, 0.5, (m, 3)) for _ in range(3)]
        nrm = unit(np.cross(v[1] - v[0], v[2] - v[0]))
        w = rng.dirichlet((1, 1, 1), m)
        on = w[:, :1] * v[0] + w[:, 1:2] * v[1] + w[:, 2:] * v[2]
        along = unit(np.cross(nrm, rng.normal(size=(m, 3))))
        d = unit(along + nrm * 10 ** rng.uniform(-6, -5, (m, 1)))
        o = (on - d * rng.uniform(2, 3, (m, 1))).astype(F)
        d = d.astype(F)
        v = [x.astype(F) for x in v]
        ok, t = _mt(*v, o, d)
        lo, hi = np.minimum(np.minimum(*v[:2]), v[2]), np.maximum(np.maximum(*v[:2]), v[2])
        with np.errstate(all="ignore"):
            entry = np.minimum((lo - o) / d, (hi - o) / d).max(1)
        pick = np.flatnonzero(ok & (t > 0.1) & (entry - t > 0.05))
        o, d, t, entry = o[pick], d[pick], t[pick], entry[pick]
        at = o + d * ((t + entry) / 2)[:, None]
        a = unit(np.cross(d, rng.normal(size=d.shape)))
        b = np.cross(d, a)
        r = F(0.01)
        small_t.append(np.stack([at + r * a, at + r * (b - a), at - r * (a + b)], 1))
        long_t.append(np.stack([x[pick] for x in v], 1))
        org.append(o)
        dirs.append(d)
    tri = np.concatenate([np.concatenate(long_t)[:n_pairs], np.concatenate(small_t)[:n_pairs]]).astype(F)
    sv, sf = scenes.displaced_icosphere(4, seed=seed)
    verts = np.concatenate([tri.reshape(-1, 3), sv.astype(F) * F(6)])
    faces = np.concatenate([np.arange(len(tri) * 3, dtype=np.uint32).reshape(-1, 3), sf.astype(np.uint32) + len(tri) * 3])
    return verts, faces, scenes._rays(np.concatenate(org)[:n_pairs], np.concatenate(dirs)[:n_pairs])
