"""The fused front of small launches (front.cu) against the oracle and against
the separate kernels.

A launch of up to 393,216 ordinals runs everything before the rasterizer in
one cooperative kernel; profiled renders keep the separate kernels, so the
two routes are compared on the same inputs: every buffer of getResources(),
the stats and the image are the same bits. The cases sit where the front
changes method: one sort tile and several, passes of 2048-item tiles (more
items than 1024 per SM), chunked passes (more than 2048 per block), no depth
pass at all (one key), one to four passes, no visible splat, an overflow."""
import importlib

import numpy as np
import pytest

import oracle
from conftest import PKG_NAME, scenes
from gpu_harness import GpuRun, assert_bit_exact, psnr

pytestmark = pytest.mark.gpu

sc = scenes()
P = importlib.import_module(PKG_NAME)

KEYS = ("visible_state", "state", "output_state", "proj_mean", "tile_counts", "visible_offsets", "depth_sorted",
        "ordered_counts", "intersection_offsets", "sorted_records", "tile_offsets", "rgba", "depth")


def cam(w=200, h=120, eye=(0.5, 1.0, 11.0), target=(0, 0, 0), **opts):
    return sc.make_frame(sc.look_at(eye, target), w, h, 55.0, 0.1, 100.0, **opts)


def slab(n, seed):
    """Splats at one view depth: every visible depth key is the same."""
    scene = sc.uniform_cloud(n, seed=seed, log_scale=(-3.0, 0.3))
    scene["means"][:, 2] = 0.0
    return scene


def dense(n, seed, log_scale=(-1.5, 0.5)):
    return sc.uniform_cloud(n, seed=seed, log_scale=log_scale)


CASES = {
    "one_splat": lambda: (sc.uniform_cloud(1, seed=1, log_scale=(-1.0, 0.1)), cam()),
    "block_edge": lambda: (sc.uniform_cloud(257, seed=2, log_scale=(-2.0, 0.5)), cam(w=33, h=17)),
    "tile_edge": lambda: (sc.uniform_cloud(1025, seed=3, log_scale=(-2.0, 0.5)), cam()),
    "one_key": lambda: (slab(3000, 4), cam(eye=(0, 0, 9.0))),
    "packed16": lambda: (sc.uniform_cloud(5000, seed=5, log_scale=(-2.4, 0.6)), cam(depth_sort_mode=1)),
    "near_and_far": lambda: (sc.uniform_cloud(20000, seed=6, extent=40.0, log_scale=(-2.0, 0.5)),
                             cam(eye=(0, 0, 0.5), target=(0, 0, 5.0))),
    "nothing_visible": lambda: (sc.uniform_cloud(3000, seed=7), cam(eye=(0, 0, 20), target=(0, 0, 40))),
    "wide_boxes": lambda: (dense(3000, 8, (0.5, 0.8)), cam(w=640, h=400)),
    "repeat_x": lambda: (sc.uniform_cloud(6000, seed=9, log_scale=(-2.4, 0.6)), cam(w=333, h=64, boundary_axis=1)),
    "many_records": lambda: (dense(40000, 10), cam(w=512, h=512)),
    "tiles_of_2048": lambda: (sc.uniform_cloud(170001, seed=16, degree=1, log_scale=(-3.8, 0.5)), cam(w=300, h=200)),
    "large_passes": lambda: (sc.uniform_cloud(200001, seed=11, log_scale=(-3.2, 0.5)), cam(w=300, h=200)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_front_equals_the_oracle_and_the_separate_kernels(name):
    scene, frame = CASES[name]()
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, "exact", capacity=max(int(o["state"][1]), 1))
    front = run.render(frame)
    assert front["launches"] == 2
    assert_bit_exact(front, o)
    run.pipe.set_profiling(True)
    separate = run.render(frame)
    assert separate["launches"] > 2
    run.pipe.set_profiling(False)
    again = run.render(frame)
    run.close()
    for k in KEYS:
        assert np.array_equal(front[k].view(np.uint32), separate[k].view(np.uint32)), k
        assert np.array_equal(front[k].view(np.uint32), again[k].view(np.uint32)), k
    assert front["stats"] == again["stats"]


@pytest.mark.parametrize("packed", [0, 1])
@pytest.mark.parametrize("n,size,log_scale", [(2047, 16, 0.0), (2048, 16, 0.0), (2049, 16, 0.0), (1000, 1024, -4.0),
                                              (2048, 1024, -4.0)])
def test_both_sides_of_the_one_block_sort(n, size, log_scale, packed):
    # All splats visible; of one tile (as many records as splats), or of 4096
    # (two passes of the tile sort, over less and more than 2048 records).
    scene = sc.uniform_cloud(n, seed=17, degree=0, log_scale=(log_scale, 0.1))
    scene["means"][:, :2] = scene["means"][:, :2] % 1.0 * 0.6 + 0.05
    frame = cam(w=size, h=size, eye=(0, 0, 20.0), depth_sort_mode=packed)
    o = oracle.render(scene, frame, 0)
    assert o["visible_state"][0] == n
    assert o["state"][0] == n if size == 16 else (o["state"][0] <= 2048) == (n == 1000)
    run = GpuRun(scene, frame, "exact", capacity=1 << 16)
    front = run.render(frame)
    run.close()
    assert front["launches"] == 2
    assert_bit_exact(front, o)


@pytest.mark.parametrize("n", [393216, 393217])
def test_both_sides_of_the_size_rule(n):
    scene, frame = sc.uniform_cloud(n, seed=12, degree=0, log_scale=(-4.0, 0.5)), cam(w=320, h=200)
    run = GpuRun(scene, frame, "exact", capacity=1 << 22)
    g = run.render(frame)
    assert (g["launches"] == 2) == (n == 393216)
    run.pipe.set_profiling(True)
    s = run.render(frame)
    run.close()
    for k in KEYS:
        assert np.array_equal(g[k].view(np.uint32), s[k].view(np.uint32)), k


def test_overflow_publishes_nothing_and_recovers():
    scene, frame = dense(4000, 13), cam()
    run = GpuRun(scene, frame, "exact", capacity=1000)
    g = run.render(frame, attempt=3, color_init=0.25)
    assert g["stats"]["overflow"] and g["stats"]["outputState"][:2] == [3, 0]
    assert (g["rgba"] == 0.25).all()
    demand = g["stats"]["requestedIntersections"]
    run.pipe.resize_intersections(demand)
    o = oracle.render(scene, frame, 0)
    assert demand == int(o["state"][1])
    assert_bit_exact(run.render(frame), o)
    run.close()


@pytest.mark.parametrize("precision", ["fp32", "half2"])
def test_batch_and_graph_of_small_views(precision):
    # Two scenes, three views, one of them a second view of its scene; the
    # front runs in the batch, in its chunks and in the graph's replays.
    import torch
    from gpu_harness import dev, pipeline_options
    a, b = (sc.uniform_cloud(n, seed=s, log_scale=(-2.6, 0.5)) for n, s in ((7000, 14), (30001, 15)))
    frames = [cam(w=160, h=90), cam(w=97, h=64, eye=(-2.0, 1.5, 10.5)), cam(w=320, h=200, eye=(3.0, 0.0, 9.0))]
    da, db = dev.DeviceScene(a), dev.DeviceScene(b)
    pipe = P.TiledGaussianPipeline(da.data(), pipeline_options(frames[0], precision, 1 << 20))
    color = [torch.zeros((f["height"], f["width"], 4), device="cuda") for f in frames]
    views = [(d.data(), P.make_camera(f), f["width"], f["height"], c.data_ptr(), 0, "rgba32f")
             for d, f, c in zip((da, db, db), frames, color)]
    images = {}

    def take(name, call):
        for c in color:
            c.zero_()
        torch.cuda.synchronize()
        call()
        torch.cuda.synchronize()
        assert not pipe.read_stats()["overflow"]
        images[name] = [c.cpu().numpy().copy() for c in color]

    take("batch", lambda: pipe.render_batch(views))
    pipe.set_profiling(True)
    take("separate", lambda: pipe.render_batch(views))
    pipe.set_profiling(False)
    pipe.set_tuning({"views_per_launch": 2})
    take("chunks", lambda: pipe.render_batch(views))
    pipe.set_tuning({"views_per_launch": 0, "work_order": 0, "tile_digit_bits": 5})
    take("tuned", lambda: pipe.render_batch(views))
    stream = torch.cuda.Stream()
    pipe.capture_graph(views, stream.cuda_stream)
    for i in range(3):
        take(f"graph{i}", lambda: pipe.launch_graph([v[1] for v in views], stream=stream.cuda_stream))
    pipe.dispose()
    for name, got in images.items():
        for g, ref, frame, scene in zip(got, images["separate"], frames, (a, b, b)):
            assert np.array_equal(g.view(np.uint32), ref.view(np.uint32)), name
    o = oracle.render(b, frames[2], 0)
    assert psnr(images["batch"][2], o["rgba"]) >= 50.0
