"""The REFERENCE walk where its box test cannot be decided by products with the
reciprocal: directions with zero, tiny and huge components, origins on box
planes, far away, infinite or not a number, flat boxes; hits bit for bit and
occlusion bits as the oracle's division test gives them."""
import numpy as np
import pytest

import scenes
from conftest import bvh2_from_export

pytestmark = pytest.mark.gpu


def _rays(n, lo, hi, planes, seed):
    rng = np.random.default_rng(seed)
    rays = scenes.incoherent_rays(lo, hi, n, seed=seed)
    o, d = rays["org"], rays["dir"]
    special = np.float32([0.0, -0.0, 1e-38, -3e-30, 1e-20, 1e30, -1e37, 1.0])
    pick = rng.random((n, 3)) < 0.25
    d[pick] = special[rng.integers(0, len(special), pick.sum())]
    on = rng.random((n, 3)) < 0.25  # origins on the planes of boxes
    axis = np.broadcast_to(np.arange(3), (n, 3))[on]
    o[on] = planes[rng.integers(0, len(planes), on.sum()), axis]
    odd = np.float32([np.nan, np.inf, -np.inf, 1e25, -1e38])
    far = rng.random(n) < 0.1
    o[far, rng.integers(0, 3, far.sum())] = odd[rng.integers(0, len(odd), far.sum())]
    return rays


@pytest.mark.parametrize("acc_name", ["BVH", "LBVH"])
@pytest.mark.parametrize("kind", ["triangles", "spheres", "flat"])
def test_reference_walk_box_decisions(engine, oracle, rqm, acc_name, kind):
    engine.configure(traversal=rqm.TRAVERSAL_REFERENCE)
    if kind == "spheres":
        rng = np.random.default_rng(4)
        sph = np.concatenate([rng.uniform(-1, 1, (3000, 3)), rng.uniform(0.01, 0.08, (3000, 1))], 1).astype(np.float32)
        scene, prims, k, pts = engine.scene_spheres(sph), np.ascontiguousarray(sph), oracle.SPHERES, sph[:, :3] + sph[:, 3:]
    else:
        v, f = scenes.displaced_icosphere(4, seed=9) if kind == "triangles" else scenes.heightfield(40, 30, amplitude=0.0, seed=3)
        prims, _, _ = oracle.tri_prims(v, f)
        scene, k, pts = engine.scene_triangles(v, f), oracle.TRIANGLES, v
    acc = engine.build(scene, getattr(rqm, acc_name))
    nodes, order, codes, root, _ = engine.export_bvh2(acc)
    tree = bvh2_from_export(oracle, nodes, order, root, codes)
    rays = _rays(20_000, pts.min(0) - 0.1, pts.max(0) + 0.1, pts, 17)
    want = oracle.trace_bvh2(k, oracle.REFERENCE, oracle.CLOSEST, tree, prims, rays)
    occ = oracle.trace_bvh2(k, oracle.REFERENCE, oracle.ANY, tree, prims, rays)
    got = engine.trace_closest(acc, rays)
    assert np.array_equal(np.ascontiguousarray(got).view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
    assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays), len(rays)), occ)
