"""Frames on both sides of the size (2^20 samples) from which the lengths of
the ray lists are read back between depths: windows of one frame, below, at
and above it, show the same pixels and count the same rays."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("acc_name,bounces", [("LBVH", 0), ("LBVH", 2), ("BVH", 1)])
def test_frame_windows_across_list_sizes(engine, rqm, acc_name, bounces):
    v, f, _ = scenes.merged_icospheres(count=40, target_tris=60_000, seed=5, levels=(3, 4))
    engine.configure(width=1056, height=1024, aa_samples=1)
    acc = engine.build(engine.scene_triangles(v, f), acc_name)
    kw = dict(eye=(0.0, -9.0, 3.0), target=(0, 0, 0), up=(0, 0, 1), fov_deg=50.0, light=(4.0, -6.0, 8.0),
              albedo=(0.7, 0.6, 0.5), ambient=0.05, mirror=0.4, bounces=bounces, seed=21)
    full, rgb, counts = engine.render(acc, rqm.make_view(**kw))  # 1,081,344 samples: lengths read back
    left, rgb_l, counts_l = engine.render(acc, rqm.make_view(window=(0, 0, 1024, 1024), **kw))  # 2^20: on the device
    right, rgb_r, counts_r = engine.render(acc, rqm.make_view(window=(1024, 0, 32, 1024), **kw))
    assert np.array_equal(full, np.concatenate([left, right], 1))
    assert np.array_equal(rgb.view(np.uint32), np.concatenate([rgb_l, rgb_r], 1).view(np.uint32))
    assert np.array_equal(np.asarray(counts), np.asarray(counts_l) + np.asarray(counts_r))
