"""Rays whose closest hit depends on the order of the walk (tests/early_hits.py):
alone, in batches of every launch form, shuffled, in many-structure queries and
in lists on the device, each ray's hit bit for bit that of the oracle's one-lane
walk, whatever rays share its warp."""
import numpy as np
import pytest

import early_hits
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
