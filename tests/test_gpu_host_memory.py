"""Device memory that a host-buffer query leaves with its context: slots as
large as the query's largest chunk, not as the largest there is."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("call", ["closest", "queries"])
def test_middle_sized_pinned_query_takes_small_slots(engine, rqm, call):
    n = 1 << 19
    v, f = scenes.displaced_icosphere(3, seed=8)
    acc = engine.build(engine.scene_triangles(v, f), rqm.LBVH)
    rays = torch.empty(n * 32, dtype=torch.uint8, pin_memory=True).numpy().view(rqm.RAY_DTYPE)
    hits = torch.empty(n * 16, dtype=torch.uint8, pin_memory=True).numpy().view(rqm.HIT_DTYPE)
    rays[:] = scenes.incoherent_rays(np.float32([-1.2] * 3), np.float32([1.2] * 3), n, seed=2)
    engine.trace_closest(acc, rays[:1000])
    free = torch.cuda.mem_get_info()[0]
    if call == "closest":
        engine.trace_closest(acc, rays, hits)
    else:
        engine.trace_queries(acc, [(rays, False, hits, -1, -1), (rays, False, hits, -1, -1)])
    # four slots of 48 bytes a ray, a chunk at most half of the query; the rest is scratch
    assert free - torch.cuda.mem_get_info()[0] < 4 * 48 * (n // 2) + (16 << 20)
    assert (hits["prim"] != rqm.MISS).any()
