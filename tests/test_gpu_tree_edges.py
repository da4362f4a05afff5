"""The LBVH at the edges of its windows (256 leaves a block): sizes around one
and several windows, runs of equal codes across them, trees as deep as the
keys allow, and batches whose scenes begin and end inside, at and across
windows, against the oracle's trees word for word."""
import numpy as np
import pytest

import scenes
from test_gpu_lbvh import _check_lbvh_against_oracle

pytestmark = pytest.mark.gpu


def _spheres(n, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "equal":
        pts = np.repeat(rng.random((1 + n // 300, 3), dtype=np.float32), 300, 0)[:n]
    elif kind == "chain":
        pts = scenes.chain_clusters(1 + int((n // 1280) ** 0.5), 64, 20)[:n]
    else:
        pts = rng.random((n, 3), dtype=np.float32)
    return np.concatenate([pts, np.full((len(pts), 1), 1e-3, np.float32)], 1).astype(np.float32)


def _codes(oracle, sph):
    lo, hi = oracle.bounds3(sph[:, :3])
    return oracle.morton_centroids(np.ascontiguousarray(sph[:, :3]), lo, hi)


@pytest.mark.parametrize("kind", ["random", "equal", "chain"])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 511, 513, 4097, 70_001])
def test_lbvh_at_window_edges(engine, oracle, rqm, n, kind):
    sph = _spheres(n, kind, n)
    acc = engine.build(engine.scene_spheres(sph), rqm.LBVH)
    if len(sph) < 2:
        nodes, order, codes, root, info = engine.export_bvh2(acc)
        assert info.n_nodes == 0 and order.tolist() == [0]
        return
    _check_lbvh_against_oracle(engine, oracle, acc, oracle.sphere_prims(sph)[0], _codes(oracle, sph))


@pytest.mark.parametrize("sizes", [[1] * 300, [256, 256, 1, 255, 2], [1, 511, 3, 513, 1, 1, 700], [2] * 129 + [3000, 5]])
def test_batched_lbvh_across_windows(engine, oracle, rqm, sizes):
    sph = [_spheres(n, "equal" if k % 3 == 1 else "random", 7 * k + n) for k, n in enumerate(sizes)]
    accs = engine.build_batched([engine.scene_spheres(x) for x in sph], rqm.LBVH)
    for x, acc in zip(sph, accs):
        if len(x) > 1:
            _check_lbvh_against_oracle(engine, oracle, acc, oracle.sphere_prims(x)[0], _codes(oracle, x))
        else:
            nodes, order, codes, root, info = engine.export_bvh2(acc)
            want = oracle.sphere_prims(x)[0].reshape(-1)
            assert info.n_nodes == 0 and order.tolist() == [0] and np.array_equal(np.ravel(root)[:6], want[:6])
