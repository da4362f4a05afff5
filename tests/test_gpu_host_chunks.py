"""Host-buffer queries of more than 2^25 rays, where the smallest chunk would
outgrow a device slot if it went by the ray count alone: the hits and bits of
the same rays queried from device memory, alone and as the last of a call."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("any_hit", [False, True])
def test_host_queries_of_more_than_two_to_the_25_rays(engine, rqm, any_hit):
    n = (1 << 25) + 513
    v, f = scenes.displaced_icosphere(4, seed=8)
    acc = engine.build(engine.scene_triangles(v, f), rqm.LBVH)
    some = scenes.incoherent_rays(np.float32([-1.2] * 3), np.float32([1.2] * 3), 1_000_003, seed=3)
    rays = np.resize(some, n)  # a length that no chunk size divides
    d = torch.from_numpy(rays.view(np.float32).reshape(n, 8)).cuda()
    if any_hit:
        want = torch.empty((n + 31) // 32, device="cuda", dtype=torch.int32)
        engine.trace_any(acc, d, want)
        got = np.empty((n + 31) // 32, np.uint32)
    else:
        want = torch.empty((n, 4), device="cuda", dtype=torch.float32)
        engine.trace_closest(acc, d, want)
        got = np.empty(n, rqm.HIT_DTYPE)
    engine.synchronize()
    want = want.cpu().numpy().view(np.uint32).reshape(-1)
    del d
    engine.trace_queries(acc, [(rays[: 1 << 22], any_hit, None, -1, -1), (rays, any_hit, got, -1, -1)])
    assert np.array_equal(got.view(np.uint32).reshape(-1), want)
    alone = engine.trace_any(acc, rays) if any_hit else engine.trace_closest(acc, rays)
    assert np.array_equal(np.ascontiguousarray(alone).view(np.uint32).reshape(-1), want)
