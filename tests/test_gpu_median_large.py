"""The median BVH of more partition tiles (1,024 positions each) than a block
adds up itself (8,192): the oracle's tree word for word."""
import numpy as np
import pytest

from test_gpu_bvh import _compare_median

pytestmark = pytest.mark.gpu


def test_median_bvh_of_more_tiles_than_a_block_adds_up(engine, oracle, rqm):
    n = 8192 * 1024 + 1
    rng = np.random.default_rng(n)
    sph = np.concatenate([rng.random((n, 3), dtype=np.float32), np.full((n, 1), 1e-3, np.float32)], 1)
    acc = engine.build(engine.scene_spheres(sph), rqm.BVH)
    aabb, cen = oracle.sphere_prims(sph)
    _compare_median(engine, oracle, rqm, acc, aabb, cen)
