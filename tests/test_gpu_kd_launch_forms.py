"""KD queries around the ray counts at which their launch changes form (one
launch whose warps have their rays by their place, up to the rays that the
resident warps hold at 32 each: seven blocks of 128 an SM for closest hits, nine
for any hit; warps taking rays from a counter above), and a million rays: every
hit and every bit as the oracle's one-lane walk."""
import numpy as np
import pytest

import scenes
from test_gpu_shared_lanes import _grazing, _u32

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _counts():
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 1
    edges = [7 * 128 * sms, 9 * 128 * sms]
    return sorted({e + d for e in edges for d in (-33, 0, 1, 33)}) + [(1 << 20) + 33]


@pytest.mark.parametrize("kind", ["closest", "any"])
def test_kd_launch_forms(engine, oracle, rqm, kind):
    v, f = scenes.heightfield(121, 77, amplitude=0.3, octaves=5, seed=5)
    prims, _, _ = oracle.tri_prims(v, f)
    acc = engine.build(engine.scene_triangles(v, f), rqm.KDTREE)
    nodes, pidx, root, _ = engine.export_kd(acc)
    counts = _counts()
    rays = _grazing(counts[-1], 17)
    query = oracle.CLOSEST if kind == "closest" else oracle.ANY
    want = oracle.trace_kd(oracle.TRIANGLES, oracle.FAST, query, oracle.Kd(nodes, pidx, root), prims, rays)
    for n in counts:
        if kind == "closest":
            assert np.array_equal(_u32(engine.trace_closest(acc, rays[:n])), _u32(want[:n])), n
        else:
            assert np.array_equal(rqm.unpack_bits(engine.trace_any(acc, rays[:n]), n), want[:n]), n
