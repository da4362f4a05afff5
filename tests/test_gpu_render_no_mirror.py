"""A frame whose surfaces mirror nothing shows the same pixels and casts the same rays whatever bounces it allows."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [160, 1100])  # list lengths on the device, read back
def test_bounces_without_a_mirror(engine, rqm, width):
    v, f = scenes.displaced_icosphere(4, seed=8)
    engine.configure(width=width, height=1000 if width > 1000 else 90, aa_samples=1)
    acc = engine.build(engine.scene_triangles(v, f), rqm.LBVH)
    kw = dict(eye=(0.0, -3.0, 1.0), target=(0, 0, 0), up=(0, 0, 1), fov_deg=50.0, light=(4.0, -6.0, 8.0),
              albedo=(0.7, 0.6, 0.5), ambient=0.05, mirror=0.0, seed=21)
    pixels, rgb, counts = engine.render(acc, rqm.make_view(bounces=0, **kw))
    assert counts[1] > 0 and counts[2] == 0
    for bounces in (1, 3):
        p, c, n = engine.render(acc, rqm.make_view(bounces=bounces, **kw))
        assert np.array_equal(p, pixels) and np.array_equal(c.view(np.uint32), rgb.view(np.uint32))
        assert list(n) == list(counts)
