"""Host-buffer queries around the sizes at which pinned arrays go chunk by
chunk (2^19 rays) and all arrays do (2^22), alone and several in one call
(closest and any hit, ordered, short and empty ones between): the hits and
bits of the same rays queried from device memory."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _pinned(a):
    t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
    v = t.numpy().view(a.dtype).reshape(a.shape)
    v[...] = a
    return v


def _rays(n, seed):
    return scenes.incoherent_rays(np.float32([-1.2] * 3), np.float32([1.2] * 3), n, seed=seed)


def _device(engine, acc, rays, any_):
    d = torch.from_numpy(rays.view(np.float32).reshape(len(rays), 8).copy()).cuda()
    if any_:
        out = torch.empty((len(rays) + 31) // 32, device="cuda", dtype=torch.int32)
        engine.trace_any(acc, d, out)
    else:
        out = torch.empty((len(rays), 4), device="cuda", dtype=torch.float32)
        engine.trace_closest(acc, d, out)
    engine.synchronize()
    return out.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("pin", [True, False])
@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19, (1 << 19) + 33, (1 << 22) + 7])
def test_host_queries_at_streaming_edges(engine, rqm, n, pin):
    v, f = scenes.displaced_icosphere(4, seed=8)
    acc = engine.build(engine.scene_triangles(v, f), rqm.LBVH)
    hold = _pinned if pin else np.array
    plan = [(n, 0, -1), (n, 1, -1), (0, 0, -1), (1000, 0, -1), (n, 0, rqm.RAY_SORT_OCTANT), (n // 2 + 1, 0, -1)]
    queries, want = [], []
    for k, (m, any_, sort) in enumerate(plan):
        rays = hold(_rays(max(m, 1), 11 * k + 1)[:m])
        out = hold(np.zeros((m + 31) // 32, np.uint32) if any_ else np.zeros(m, rqm.HIT_DTYPE))
        queries.append((rays, any_, out, sort, -1))
        want.append(_device(engine, acc, rays, any_).reshape(-1) if m else np.zeros(0, np.uint32))
    for _ in range(2):  # the slots in another rotation the second time
        engine.trace_queries(acc, queries)
        for q, w in zip(queries, want):
            assert np.array_equal(np.ascontiguousarray(q[2]).view(np.uint32).reshape(-1), w)
            q[2].view(np.uint8)[...] = 0
    single = engine.trace_closest(acc, queries[0][0])
    assert np.array_equal(np.ascontiguousarray(single).view(np.uint32).reshape(-1), want[0])
