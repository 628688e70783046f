"""Batches of many views of one small scene in the fused front: the views share
the scene's projection blocks, every later stage has all their ordinals. The
same bits as the separate kernels, view by view the oracle's."""
import numpy as np
import pytest

import oracle
from conftest import pkg, scenes
from gpu_harness import dev, pipeline_options

pytestmark = pytest.mark.gpu

sc = scenes()


@pytest.mark.parametrize("views,n,degree", [(12, 32000, 1), (150, 2300, 0), (33, 257, 2)])
def test_many_views_of_one_scene(views, n, degree):
    import torch
    P = pkg()
    scene = sc.uniform_cloud(n, seed=41, degree=degree, log_scale=(-3.2, 0.5))
    frames = [sc.make_frame(sc.look_at((11.0 * np.sin(a), 1.0, 11.0 * np.cos(a)), (0, 0, 0)), 96 + 8 * (i % 3), 64,
                            55.0, 0.1, 100.0) for i, a in enumerate(np.linspace(0.0, 6.0, views))]
    ds = dev.DeviceScene(scene)
    pipe = P.TiledGaussianPipeline(ds.data(), pipeline_options(frames[0], "exact", 1 << 21))
    color = [torch.zeros((f["height"], f["width"], 4), device="cuda") for f in frames]
    batch = [(ds.data(), P.make_camera(f), f["width"], f["height"], c.data_ptr(), 0, "rgba32f")
             for f, c in zip(frames, color)]

    def take():
        for c in color:
            c.zero_()
        torch.cuda.synchronize()
        pipe.render_batch(batch)
        stats = pipe.read_stats()
        assert not stats["overflow"]
        r = pipe.get_resources()
        V, cnt = stats["visibleGaussianCount"], stats["intersectionCount"]
        buffers = [dev.to_numpy(p, (k,)) for p, k in (
            (r.depth_sorted_keys, V), (r.depth_sorted_ids, V), (r.depth_ordered_tile_counts, V),
            (r.intersection_offsets, V), (r.sorted_tile_ids, cnt), (r.sorted_gaussian_ids, cnt),
            (r.tile_offsets, pipe.batch_layout()[1][-1] + 1), (r.visible_offsets, pipe.batch_layout()[0][-1]))]
        return stats, [b.copy() for b in buffers] + [c.cpu().numpy().view(np.uint32) for c in color]

    stats, front = take()
    assert pipe.last_launch_count() == 2
    pipe.set_profiling(True)
    same, separate = take()
    assert pipe.last_launch_count() > 2
    pipe.dispose()
    assert stats == same
    if (views, n) == (12, 32000):  # more than a tile of 2048 for each of 152 blocks
        assert stats["visibleGaussianCount"] > 311296
    for a, b in zip(front, separate):
        assert np.array_equal(a, b)
    for i in (0, views // 2, views - 1):
        o = oracle.render(scene, frames[i], 0)
        assert np.array_equal(front[8 + i], o["rgba"].view(np.uint32))
