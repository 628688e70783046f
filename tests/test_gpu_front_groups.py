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


@pytest.mark.parametrize("precision,axis", [("exact", 0), ("half2", 0), ("half2", 1)])
def test_groups_of_a_large_scene_beside_spread_views_of_a_small_one(precision, axis):
    # Ten views: five and two of a scene that fills the SMs by itself (a group
    # each), between them three of a small one (each its own group). Every
    # view's image is that of its own render, in the batch and in a graph.
    import torch
    P = pkg()
    a, b = (sc.uniform_cloud(n, seed=s, degree=d, log_scale=(-3.0, 0.5)) for n, s, d in ((160001, 42, 1), (3001, 43, 3)))
    da, db = dev.DeviceScene(a), dev.DeviceScene(b)
    frames = [sc.make_frame(sc.look_at((11.0 * np.sin(i), 1.0, 11.0 * np.cos(i)), (0, 0, 0)), 128 - 8 * (i % 2), 72,
                            55.0, 0.1, 100.0, boundary_axis=axis) for i in range(10)]
    owner = [da] * 5 + [db] * 3 + [da] * 2
    color = [torch.zeros((f["height"], f["width"], 4), device="cuda") for f in frames]
    views = [(d.data(), P.make_camera(f), f["width"], f["height"], c.data_ptr(), 0, "rgba32f")
             for d, f, c in zip(owner, frames, color)]
    pipe = P.TiledGaussianPipeline(da.data(), pipeline_options(frames[0], precision, 1 << 22))

    def take(call):
        for c in color:
            c.zero_()
        torch.cuda.synchronize()
        call()
        assert not pipe.read_stats()["overflow"]
        return [c.cpu().numpy().view(np.uint32).copy() for c in color]

    images = [take(lambda: pipe.render_batch(views))]
    stream = torch.cuda.Stream()
    pipe.capture_graph(views, stream.cuda_stream)
    images += [take(lambda: pipe.launch_graph([v[1] for v in views], stream=stream.cuda_stream)) for _ in range(2)]
    for i, v in enumerate(views):
        alone = take(lambda: pipe.render_batch([v]))[i]
        assert alone.any()
        for got in images:
            assert np.array_equal(got[i], alone), i
    pipe.dispose()
