"""Queries on spheres, whose closest hits keep their lane: in one launch and
from the counter, and in many-structure queries whose warps take 64 rays at a
time, around a warp's rays and a turn's, against the oracle's walk bit for bit."""
import numpy as np
import pytest

import scenes
from conftest import bvh2_from_export

pytestmark = pytest.mark.gpu


def _u32(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _spheres(n, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.uniform(-1, 1, (n, 3)), rng.uniform(0.01, 0.06, (n, 1))], 1).astype(np.float32)


def _rays(n, seed):
    return scenes.incoherent_rays(np.float32([-1.3] * 3), np.float32([1.3] * 3), n, seed=seed)


def _want(engine, oracle, acc, sph, rays):
    nodes, order, codes, root, _ = engine.export_bvh2(acc)
    tree = bvh2_from_export(oracle, nodes, order, root, codes)
    return [oracle.trace_bvh2(oracle.SPHERES, oracle.FAST, q, tree, sph, rays) for q in (oracle.CLOSEST, oracle.ANY)]


@pytest.mark.parametrize("n_rays", [1, 1000, 300_003])
@pytest.mark.parametrize("structure", ["LBVH", "BVH"])
def test_sphere_walks_one_structure(engine, oracle, rqm, structure, n_rays):
    sph = _spheres(3000, 1)
    acc = engine.build(engine.scene_spheres(sph), getattr(rqm, structure))
    rays = _rays(n_rays, 2)
    hits, occ = _want(engine, oracle, acc, sph, rays)
    assert np.array_equal(_u32(engine.trace_closest(acc, rays)), _u32(hits))
    assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays), n_rays), occ)


@pytest.mark.parametrize("counts", [[1], [31, 2], [64], [65, 1, 63], [37, 4000, 100, 64 * 19 + 33]])
def test_sphere_walks_many_structures(engine, oracle, rqm, counts):
    sph = [_spheres(50 + 700 * k, 5 + k) for k in range(len(counts))]
    accs = engine.build_batched([engine.scene_spheres(s) for s in sph], rqm.LBVH)
    rays = [_rays(n, 20 + k) for k, n in enumerate(counts)]
    offs = np.concatenate([[0], np.cumsum(counts)])
    hits = engine.trace_batched(accs, np.concatenate(rays), offs)
    bits = rqm.unpack_bits(engine.trace_batched(accs, np.concatenate(rays), offs, any_hit=True), int(offs[-1]))
    for k, s in enumerate(sph):
        want, occ = _want(engine, oracle, accs[k], s, rays[k])
        assert np.array_equal(_u32(hits[offs[k]:offs[k + 1]]), _u32(want)), k
        assert np.array_equal(bits[offs[k]:offs[k + 1]], occ), k
