"""The KD builder at the edges of its passes: cost runs (128 edges), node
tiles (256), side tiles (1,024 refs), partition tiles (2,048 edges) and the
line between counts a block adds up itself and the scanned ones (1,024 tiles
a list: 1,048,576 primitives), with runs of equal planes across them and
rebuilds that reuse larger buffers, against the oracle's tree word for word."""
import numpy as np
import pytest

from test_gpu_kd import _check_nodes

pytestmark = pytest.mark.gpu


def _spheres(n, seed):
    rng = np.random.default_rng(seed)
    sph = np.concatenate([rng.random((n, 3), dtype=np.float32), rng.uniform(1e-3, 2e-2, (n, 1))], 1).astype(np.float32)
    sph[rng.random(n) < 0.15] = sph[0]
    sph[:, 2] = np.round(sph[:, 2] * 16) / 16
    return sph


def _check(engine, oracle, rqm, sph, depth=-1):
    engine.configure(kd_max_depth=depth)
    acc = engine.build(engine.scene_spheres(sph), rqm.KDTREE)
    ref = oracle.build_kd(oracle.sphere_prims(sph)[0], depth)
    for _ in range(2):
        nodes, pidx, _, _ = engine.export_kd(acc)
        _check_nodes(nodes, pidx, ref.nodes, ref.prim_idx)
        acc.rebuild()
    acc.close()
    engine.configure(kd_max_depth=-1)


@pytest.mark.parametrize("n", [1, 2, 5, 6, 63, 64, 65, 511, 512, 1023, 1024, 1025, 5000, 20_001])
def test_kd_at_pass_edges(engine, oracle, rqm, n):
    _check(engine, oracle, rqm, _spheres(n, n))


@pytest.mark.parametrize("n", [1 << 20, (1 << 20) + 1])
def test_kd_at_the_scanned_partition_line(engine, oracle, rqm, n):
    _check(engine, oracle, rqm, _spheres(n, 3), depth=3)


def test_kd_small_after_large(engine, oracle, rqm):
    """One context's buffers, grown by a larger tree, then a small one and the larger again."""
    for n in (30_000, 200, 30_000):
        _check(engine, oracle, rqm, _spheres(n, 5))
