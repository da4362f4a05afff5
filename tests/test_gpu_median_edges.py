"""The median BVH at the edges of its parts: the in-block span (1,024
primitives), the partition's tiles (1,024 positions), a level's one-block pass
(1,024 segments a round, from about a million primitives on), runs of equal
centroids across them, against the oracle's tree word for word."""
import numpy as np
import pytest

from test_gpu_bvh import _compare_median

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 1023, 1024, 1025, 2047, 2049, 4097, 65_537, 2_200_001])
def test_median_bvh_at_part_edges(engine, oracle, rqm, n):
    rng = np.random.default_rng(n)
    sph = np.concatenate([rng.random((n, 3), dtype=np.float32), np.full((n, 1), 1e-3, np.float32)], 1)
    if n < 100_000:
        sph[rng.random(n) < 0.2] = sph[0]  # equal centroids: ties by id, leaves of several primitives
        sph[:, 1] = np.round(sph[:, 1] * 8) / 8  # and equal coordinates along one axis
    acc = engine.build(engine.scene_spheres(sph), rqm.BVH)
    aabb, cen = oracle.sphere_prims(sph)
    _compare_median(engine, oracle, rqm, acc, aabb, cen)
