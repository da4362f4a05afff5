"""Rays of a warp that share its lanes: long grazing rays over a terrain (so
that subtrees move between lanes from the first rounds on), at ray counts
around one ray a warp, a part of a warp, one full grid and several, closest
and any hit, in one-structure and many-structure queries: every hit bit for
bit, and every occlusion bit, as the oracle's one-lane walk of the exported
structure."""
import numpy as np
import pytest

import scenes
from conftest import bvh2_from_export

pytestmark = pytest.mark.gpu


def _u32(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _grazing(n, seed):
    """Origins at the border of [-1, 1]^2 near the surface, directions almost level."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 2 * np.pi, n)
    o = np.stack([1.2 * np.cos(a), 1.2 * np.sin(a), rng.uniform(-0.1, 0.3, n)], 1)
    t = np.stack([rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), rng.uniform(-0.2, 0.3, n)], 1)
    d = t - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return scenes._rays(o.astype(np.float32), d.astype(np.float32))


@pytest.fixture(scope="module")
def terrain():
    return scenes.heightfield(121, 77, amplitude=0.3, octaves=5, seed=5)


def _oracle_tree(engine, oracle, acc):
    nodes, order, codes, root, _ = engine.export_bvh2(acc)
    return bvh2_from_export(oracle, nodes, order, root, codes)


@pytest.mark.parametrize("n_rays", [1, 2, 33, 900, 5000, 50_000, 250_003])
@pytest.mark.parametrize("acc_name", ["LBVH", "BVH"])
def test_shared_lanes_one_structure(engine, oracle, rqm, terrain, acc_name, n_rays):
    v, f = terrain
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), getattr(rqm, acc_name))
    tree = _oracle_tree(engine, oracle, acc)
    rays = _grazing(n_rays, 40 + n_rays)
    want = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, tree, prims, rays)
    occ = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.ANY, tree, prims, rays)
    assert 0.05 < occ.mean() < 0.999 or n_rays < 100
    assert np.array_equal(_u32(engine.trace_closest(acc, rays)), _u32(want))
    assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays), n_rays), occ)


def test_shared_lanes_rays_with_a_zero_direction_component(engine, oracle, rqm, terrain):
    """Rays set aside for the exact box test among rays that share lanes, fewer than a grid."""
    v, f = terrain
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), rqm.LBVH)
    tree = _oracle_tree(engine, oracle, acc)
    rays = _grazing(1500, 3)
    rays["dir"][::7] = (0.0, 0.0, -1.0)
    rays["org"][::7, 2] = 2.0
    want = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, tree, prims, rays)
    occ = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.ANY, tree, prims, rays)
    assert np.array_equal(_u32(engine.trace_closest(acc, rays)), _u32(want))
    assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays), len(rays)), occ)


def test_shared_lanes_rays_without_an_end(engine, oracle, rqm, terrain):
    """tmax infinite or not a number, tmin above tmax, among rays that share lanes: the oracle's bits."""
    v, f = terrain
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), rqm.LBVH)
    tree = _oracle_tree(engine, oracle, acc)
    rays = _grazing(5000, 13)
    rays["tmax"][::5] = np.nan
    rays["tmax"][1::7] = np.inf
    rays["tmax"][2::11] = -1.0
    want = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, tree, prims, rays)
    occ = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.ANY, tree, prims, rays)
    assert np.array_equal(_u32(engine.trace_closest(acc, rays)), _u32(want))
    assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays), len(rays)), occ)


def test_shared_lanes_many_structures(engine, oracle, rqm, terrain):
    """Warps whose rays belong to several structures of different sizes."""
    meshes = [terrain, scenes.displaced_icosphere(2, seed=4), scenes.heightfield(9, 7, seed=6), terrain]
    counts = [37, 5, 11, 4000]
    accs = engine.build_batched([engine.scene_triangles(v, f) for v, f in meshes], rqm.LBVH)
    rays = [_grazing(n, 60 + k) for k, n in enumerate(counts)]
    rays[3]["dir"][5] = (1.0, 0.0, 0.0)  # one ray for the exact box test
    offs = np.concatenate([[0], np.cumsum(counts)])
    hits = engine.trace_batched(accs, np.concatenate(rays), offs)
    bits = rqm.unpack_bits(engine.trace_batched(accs, np.concatenate(rays), offs, any_hit=True), int(offs[-1]))
    for k, (v, f) in enumerate(meshes):
        prims, _, _ = oracle.tri_prims(v, f)
        tree = _oracle_tree(engine, oracle, accs[k])
        want = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, tree, prims, rays[k])
        occ = oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.ANY, tree, prims, rays[k])
        assert np.array_equal(_u32(hits[offs[k]:offs[k + 1]]), _u32(want)), k
        assert np.array_equal(bits[offs[k]:offs[k + 1]], occ), k


def _kd_check(engine, oracle, rqm, kind, scene, prims, rays):
    acc = engine.build(scene, rqm.KDTREE)
    nodes, pidx, root, _ = engine.export_kd(acc)
    kd = oracle.Kd(nodes, pidx, root)
    want = oracle.trace_kd(kind, oracle.FAST, oracle.CLOSEST, kd, prims, rays)
    occ = oracle.trace_kd(kind, oracle.FAST, oracle.ANY, kd, prims, rays)
    assert np.array_equal(_u32(engine.trace_closest(acc, rays)), _u32(want))
    assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays), len(rays)), occ)
    return want


@pytest.mark.parametrize("n_rays", [1, 33, 900, 50_000, 250_003])
def test_shared_lanes_kd(engine, oracle, rqm, terrain, n_rays):
    """The first closest hit in the walk's order, whichever lane finds it."""
    v, f = terrain
    prims, _, _ = oracle.tri_prims(v, f)
    _kd_check(engine, oracle, rqm, oracle.TRIANGLES, engine.scene_triangles(v, f), prims, _grazing(n_rays, 80 + n_rays))


def test_shared_lanes_kd_any_hit_million_rays(engine, oracle, rqm, terrain):
    """A launch of more than 2^20 rays gives the bits of its parts."""
    v, f = terrain
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), rqm.KDTREE)
    rays = _grazing((1 << 20) + 33, 7)
    bits = rqm.unpack_bits(engine.trace_any(acc, rays), len(rays))
    below = rqm.unpack_bits(engine.trace_any(acc, rays[:1 << 20]), 1 << 20)
    assert np.array_equal(bits[:1 << 20], below)


@pytest.mark.parametrize("depth", [1, 4, 9])
@pytest.mark.parametrize("n_rays", [1, 33, 20_001])
def test_shared_lanes_kd_long_leaves(engine, oracle, rqm, terrain, n_rays, depth):
    """Leaves of dozens to thousands of primitives, each triangle there three times: equal distances within and across
    batches of 32 go to the first of the leaf's list."""
    v, f = terrain
    f = np.concatenate([f[: len(f) // 8]] * 3)
    engine.configure(kd_max_depth=depth)
    prims, _, _ = oracle.tri_prims(v, f)
    _kd_check(engine, oracle, rqm, oracle.TRIANGLES, engine.scene_triangles(v, f), prims, _grazing(n_rays, 90 + n_rays))


@pytest.mark.parametrize("n_rays", [700, 100_003])
def test_shared_lanes_kd_small_distant_spheres(engine, oracle, rqm, n_rays):
    """Spheres whose hit distances cancel: hits before their leaf's interval, equal distances, rays in doubt."""
    rng = np.random.default_rng(9)
    p = rng.normal(size=(5000, 3))
    p /= np.linalg.norm(p, axis=1, keepdims=True)
    sph = np.concatenate([p * 3.6 + np.array([-2.0, 5.0, -58.0]), np.full((5000, 1), 0.05)], 1).astype(np.float32)
    t = p[rng.integers(0, 5000, n_rays)] * rng.uniform(0.2, 1.02, (n_rays, 1)) * 3.6 + np.array([-2.0, 5.0, -58.0])
    d = t / np.linalg.norm(t, axis=1, keepdims=True)
    rays = scenes._rays(np.zeros((n_rays, 3), np.float32), d.astype(np.float32))
    want = _kd_check(engine, oracle, rqm, oracle.SPHERES, engine.scene_spheres(sph), sph, rays)
    assert (want["prim"] != rqm.MISS).mean() > 0.2
