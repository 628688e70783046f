"""Tiles of 8 and 32 pixels in the separate kernels: small batches run the fused
front there, profiled ones do not. Every buffer and the EXACT image are the same
bits on both routes; the image is that of 16-pixel tiles, whose buffers the
oracle checks elsewhere."""
import numpy as np
import pytest

from conftest import pkg, scenes
from gpu_harness import dev, pipeline_options
from test_gpu_half2_needles import needle_cloud

pytestmark = pytest.mark.gpu

sc = scenes()


CASES = {
    "wide": (sc.uniform_cloud(3000, seed=51, log_scale=(0.2, 0.8)), {}),
    "needles": (needle_cloud(6000, seed=52), {}),
    "fp64": (needle_cloud(6000, seed=53), {"projection_precision": "fp64"}),
    "repeat_x": (sc.uniform_cloud(6000, seed=54, log_scale=(-1.6, 0.6)), {"boundary_axis": 1}),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_both_routes_at_every_tile_size(name):
    import torch
    P = pkg()
    scene, options = CASES[name]
    ds = dev.DeviceScene(scene)
    frames = [sc.make_frame(sc.look_at(eye, (0, 0, 0)), w, h, 55.0, 0.1, 100.0, **options)
              for eye, w, h in (((0.5, 1.0, 11.0), 640, 400), ((-2.0, 1.5, 9.0), 321, 203))]
    pipe = P.TiledGaussianPipeline(ds.data(), pipeline_options(frames[0], "exact", 1 << 24))
    color = [torch.zeros((f["height"], f["width"], 4), device="cuda") for f in frames]
    views = [(ds.data(), P.make_camera(f), f["width"], f["height"], c.data_ptr(), 0, "rgba32f")
             for f, c in zip(frames, color)]

    def take(tile, profiled):
        pipe.set_tuning({"tile_size": tile})
        pipe.set_profiling(profiled)
        for c in color:
            c.zero_()
        torch.cuda.synchronize()
        pipe.render_batch(views)
        stats = pipe.read_stats()
        assert not stats["overflow"]
        assert (pipe.last_launch_count() == 2) == (not profiled and name != "fp64")
        r = pipe.get_resources()
        item, tiles = (b[-1] for b in pipe.batch_layout())
        V, cnt = stats["visibleGaussianCount"], stats["intersectionCount"]
        got = [dev.to_numpy(p, (k,)).copy() for p, k in (
            (r.tile_counts, item), (r.visible_offsets, item), (r.depth_sorted_keys, V), (r.depth_sorted_ids, V),
            (r.depth_ordered_tile_counts, V), (r.intersection_offsets, V), (r.sorted_tile_ids, cnt),
            (r.sorted_gaussian_ids, cnt), (r.tile_offsets, tiles + 1))]
        return got, [c.cpu().numpy().view(np.uint32).copy() for c in color]

    image = take(16, False)[1]
    for tile in (8, 16, 32):
        front, a = take(tile, False)
        separate, b = take(tile, True)
        for x, y in zip(front + a, separate + b):
            assert np.array_equal(x, y), tile
        for x, y in zip(a, image):
            assert np.array_equal(x, y), tile
        assert len(front[6]) > 0
    pipe.dispose()
