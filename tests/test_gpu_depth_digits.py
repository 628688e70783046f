"""The digits of the depth sort's separate kernels against the oracle.

The separate kernels sort the float32 keys by 9-bit digits of their distance
from the nearest near plane, in as few passes as the batch's depth range
needs, if those are fewer than the four of 8 bits. The ranges sit on
both sides of each number of passes (9, 18 and 27 bits); the keys and ids come
out the same for all of them. Profiled renders keep the separate kernels at
these sizes."""
import importlib

import numpy as np
import pytest

import oracle
from conftest import PKG_NAME, scenes
from gpu_harness import GpuRun, assert_bit_exact

pytestmark = pytest.mark.gpu

sc = scenes()
P = importlib.import_module(PKG_NAME)


def bits_of(near, far):
    low, high = (int(np.float32(x).view(np.uint32)) for x in (near, far))
    return max(1, (high - low).bit_length())


def above(x, ulps):
    return float((np.float32(x).view(np.uint32) + np.uint32(ulps)).view(np.float32))


# near, far, bits of their difference, passes
RANGES = [(0.1, 1000.0, 27, 3), (1.0, above(1.0, (1 << 27) - 1), 27, 3), (1.0, above(1.0, 1 << 27), 28, 4),
          (0.0, 100.0, 31, 4), (-0.0, 50.0, 31, 4), (0.5, 3.0e38, 31, 4), (8.0, 14.0, 23, 3),
          (10.5, above(10.5, (1 << 18) - 1), 18, 2), (10.5, above(10.5, 1 << 18), 19, 3),
          (11.0, above(11.0, 511), 9, 1), (11.0, above(11.0, 512), 10, 2)]


@pytest.mark.parametrize("near,far,bits,passes", RANGES)
@pytest.mark.parametrize("n", [1, 4097, 30001])
def test_every_number_of_passes(n, near, far, bits, passes):
    assert bits_of(abs(near), far) == bits
    scene = sc.uniform_cloud(n, seed=n, degree=0, log_scale=(-3.0, 0.5))
    if n > 1:
        # A seventh of the splats some units in the last place beyond 11.0.
        scene["means"][::7, 2] = -(np.arange(len(scene["means"][::7])) % 600) * np.float32(2.0**-20)
    frame = sc.make_frame(sc.look_at((0.0, 0.0, 11.0), (0.0, 0.0, 0.0)), 200, 120, 55.0, 0.1, 100.0, depth_encoding=1)
    frame.update(near=near, far=far)
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, "exact", capacity=max(int(o["state"][1]), 1))
    run.pipe.set_profiling(True)
    g = run.render(frame)
    assert_bit_exact(g, o)
    everything = dict(frame, near=0.0, far=3.0e38)  # no range left: four passes
    launches = run.render(everything)["launches"]
    run.close()
    assert launches - g["launches"] == 2 * (4 - passes)


def test_views_with_their_own_ranges():
    # The batch's keys span the nearest near to the farthest far plane.
    import torch
    from gpu_harness import dev, pipeline_options
    scene = sc.uniform_cloud(9001, seed=5, log_scale=(-2.6, 0.5))
    view = sc.look_at((0.5, 1.0, 11.0), (0.0, 0.0, 0.0))
    frames = [sc.make_frame(view, 160, 90, 55.0, near, far) for near, far in ((9.0, 12.0), (2.0, 10.0), (11.0, 90.0))]
    data = dev.DeviceScene(scene)
    pipe = P.TiledGaussianPipeline(data.data(), pipeline_options(frames[0], "exact", 1 << 20))
    color = [torch.zeros((90, 160, 4), device="cuda") for _ in frames]
    views = [(data.data(), P.make_camera(f), 160, 90, c.data_ptr(), 0, "rgba32f") for f, c in zip(frames, color)]
    pipe.set_profiling(True)
    pipe.render_batch(views)
    torch.cuda.synchronize()
    assert not pipe.read_stats()["overflow"]
    got = [c.cpu().numpy().copy() for c in color]
    pipe.dispose()
    for g, frame in zip(got, frames):
        assert np.array_equal(g.view(np.uint32), oracle.render(scene, frame, 0)["rgba"].view(np.uint32))


def test_a_captured_graph_takes_every_range():
    # Captured with planes 10 and 12 away, replayed with planes at 0 and 1e6.
    import torch
    from gpu_harness import dev, pipeline_options
    n = 400_001  # beyond the fused front
    scene = sc.uniform_cloud(n, seed=6, degree=0, log_scale=(-4.0, 0.5))
    view = sc.look_at((0.0, 0.0, 11.0), (0.0, 0.0, 0.0))
    captured = sc.make_frame(view, 160, 90, 55.0, 10.0, 12.0)
    wide = dict(captured, near=0.0, far=1.0e6)
    data = dev.DeviceScene(scene)
    pipe = P.TiledGaussianPipeline(data.data(), pipeline_options(captured, "exact", 1 << 21))
    color = torch.zeros((90, 160, 4), device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    images = []
    for frame in (captured, wide):
        pipe.render_batch([(data.data(), P.make_camera(frame), 160, 90, color.data_ptr(), 0, "rgba32f")])
        torch.cuda.synchronize()
        images.append(color.cpu().numpy().copy())
    pipe.capture_graph([(data.data(), P.make_camera(captured), 160, 90, color.data_ptr(), 0, "rgba32f")],
                       stream.cuda_stream)
    for frame, image in ((wide, images[1]), (captured, images[0]), (wide, images[1])):
        pipe.launch_graph([P.make_camera(frame)], stream=stream.cuda_stream)
        stream.synchronize()
        assert not pipe.read_stats()["overflow"]
        assert np.array_equal(color.cpu().numpy().view(np.uint32), image.view(np.uint32))
    pipe.dispose()
    assert not np.array_equal(images[0], images[1])
