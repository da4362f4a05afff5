"""Rays whose closest hit depends on the order of the walk (tests/early_hits.py):
alone, in batches of every launch form, shuffled, in many-structure queries and
in lists on the device, each ray's hit bit for bit that of the oracle's one-lane
walk, whatever rays share its warp."""
import numpy as np
import pytest

import early_hits
import scenes
from conftest import bvh2_from_export

pytestmark = pytest.mark.gpu


def _u32(a):
    return np.ascontiguousarray(a).view(np.uint32).reshape(-1, 4)


def _want(engine, oracle, acc, prims, rays):
    nodes, order, codes, root, _ = engine.export_bvh2(acc)
    tree = bvh2_from_export(oracle, nodes, order, root, codes)
    return _u32(oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, tree, prims, rays))


@pytest.mark.parametrize("structure", ["LBVH", "BVH"])
def test_early_hits_one_structure(engine, oracle, rqm, structure):
    v, f, rays = early_hits.scene_and_rays(1500, 1)
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), getattr(rqm, structure))
    want = _want(engine, oracle, acc, prims, rays)
    brute = oracle.trace_brute(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, prims, rays)
    assert (want[:, 1] != brute["prim"]).sum() > 50  # the order decides
    for k in range(20):
        assert np.array_equal(_u32(engine.trace_closest(acc, rays[k:k + 1])), want[k:k + 1])
    rng = np.random.default_rng(2)
    for n in (33, 700, 1500, 40_000, 300_003):
        pick = rng.integers(0, len(rays), n)
        assert np.array_equal(_u32(engine.trace_closest(acc, rays[pick])), want[pick]), n


def test_early_hits_many_structures(engine, oracle, rqm):
    parts = [early_hits.scene_and_rays(n, 10 + k) for k, n in enumerate((5, 400, 37, 900))]
    accs = engine.build_batched([engine.scene_triangles(v, f) for v, f, _ in parts], rqm.LBVH)
    offs = np.concatenate([[0], np.cumsum([len(r) for _, _, r in parts])])
    hits = _u32(engine.trace_batched(accs, np.concatenate([r for _, _, r in parts]), offs))
    for k, (v, f, rays) in enumerate(parts):
        prims, _, _ = oracle.tri_prims(v, f)
        assert np.array_equal(hits[offs[k]:offs[k + 1]], _want(engine, oracle, accs[k], prims, rays)), k


def test_imported_boxes_that_do_not_hold_their_primitives(engine, oracle, rqm):
    """Two surfaces, one below the other; leaf boxes of the upper one sunk below the lower one: hits from above lie before
    the box they are found through, and a hit on the lower surface culls that box."""
    v, f = scenes.heightfield(61, 47, amplitude=0.3, octaves=4, seed=5)
    n = len(f)
    v2, f2 = np.concatenate([v, v - np.float32([0, 0, 0.05])]), np.concatenate([f, f + len(v)])
    scene = engine.scene_triangles(v2, f2)
    prims, _, _ = oracle.tri_prims(v2, f2)
    nodes, order, codes, root, _ = engine.export_bvh2(engine.build(scene, rqm.LBVH))
    nodes = np.array(nodes, np.float32).reshape(-1, 16)
    links = nodes[:, 12:].view(np.int32)
    rng = np.random.default_rng(4)
    for side in (0, 1):
        leaf = (links[:, side] < 0) & (rng.random(len(nodes)) < 0.5)
        leaf[leaf] = np.asarray(order)[~links[leaf, side]] < n
        for lo, hi in ((0, 1), (2, 3)):
            nodes[leaf, 4 * side + lo] -= 0.1
            nodes[leaf, 4 * side + hi] += 0.1
        nodes[leaf, 9 + 2 * side] = nodes[leaf, 8 + 2 * side] - np.float32(0.1)
        nodes[leaf, 8 + 2 * side] -= np.float32(2)
    box = np.float32([-9, -9, -9, 9, 9, 9])
    acc = engine.import_bvh2(scene, nodes, order, box)
    o = rng.uniform([-1, -1, 1], [1, 1, 2], (30_000, 3)).astype(np.float32)
    d = rng.uniform([-1, -1, 0], [1, 1, 0], (30_000, 3)).astype(np.float32) - o
    rays = scenes._rays(o, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32))
    want = _u32(oracle.trace_bvh2(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST,
                                  bvh2_from_export(oracle, nodes, order, box), prims, rays))
    assert 0.1 < (want[:, 1] < n).mean() < 0.9
    for m in (1, 33, 700, 30_000):
        assert np.array_equal(_u32(engine.trace_closest(acc, rays[:m])), want[:m]), m
    pick = rng.integers(0, len(rays), 300_003)
    assert np.array_equal(_u32(engine.trace_closest(acc, rays[pick])), want[pick])
    plain = engine.build(scene, rqm.LBVH)
    offs = np.array([0, len(rays), len(rays) + 900])
    assert np.array_equal(_u32(engine.trace_batched([acc, plain], np.concatenate([rays, rays[:900]]), offs))[:len(rays)], want)


def test_early_hits_kd(engine, oracle, rqm):
    v, f, rays = early_hits.scene_and_rays(1500, 1)
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), rqm.KDTREE)
    nodes, pidx, root, _ = engine.export_kd(acc)
    want = _u32(oracle.trace_kd(oracle.TRIANGLES, oracle.FAST, oracle.CLOSEST, oracle.Kd(nodes, pidx, root), prims, rays))
    for k in range(20):
        assert np.array_equal(_u32(engine.trace_closest(acc, rays[k:k + 1])), want[k:k + 1])
    rng = np.random.default_rng(2)
    for n in (33, 700, 1500, 40_000, 300_003):
        pick = rng.integers(0, len(rays), n)
        assert np.array_equal(_u32(engine.trace_closest(acc, rays[pick])), want[pick]), n
