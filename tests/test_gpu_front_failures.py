"""The fused front of small launches where its cooperative launch is refused
and where its blocks wait in vain, made to happen without a GPU fault.

* A refused launch (an error code on the host, as on a stream that may use only
  a part of the device's SMs): the separate kernels render the frame. Nothing
  else may read the workspaces, which hold no frame yet.
* A barrier that runs out: the block that compacts the first splats leaves, the
  others give up after the set number of polls, the frame reports
  GS3D_ERROR_DEVICE_TIMEOUT and writes no pixel, and the same pipeline renders
  the next frame bit-exact. A limit too short for the front's barriers keeps
  the separate kernels, whose waits it bounds (test_gpu_failures.py).
"""
import importlib

import numpy as np
import pytest

import oracle
from conftest import PKG_NAME, scenes
from gpu_harness import GpuRun, assert_bit_exact

pytestmark = pytest.mark.gpu

sc = scenes()
P = importlib.import_module(PKG_NAME)


def case(n=6000, seed=91):
    scene = sc.uniform_cloud(n, seed=seed, log_scale=(-2.4, 0.6))
    return scene, sc.make_frame(sc.look_at((0.5, 1.0, 11.0), (0, 0, 0)), 200, 120, 55.0, 0.1, 100.0)


def test_refused_front_renders_by_the_separate_kernels():
    scene, frame = case()
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, "exact", capacity=int(o["state"][1]) + 256)
    run.pipe.debug_refuse_front()
    first = run.render(frame)  # a new pipeline's first frame: every workspace is as allocated
    assert first["launches"] > 2
    assert_bit_exact(first, o)
    # The refusal was of that launch alone.
    again = run.render(frame)
    assert again["launches"] == 2
    assert_bit_exact(again, o)
    run.close()


def test_refused_front_in_a_captured_graph():
    import torch
    scene, frame = case(seed=92)
    run = GpuRun(scene, frame, "exact", capacity=1 << 18)
    ref = run.render(frame)
    H, W = int(frame["height"]), int(frame["width"])
    color = torch.zeros((H, W, 4), device="cuda")
    cam = P.make_camera(frame)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    run.pipe.debug_refuse_front()
    run.pipe.capture_graph([(run.ds.data(), cam, W, H, color.data_ptr(), 0, "rgba32f")], stream.cuda_stream)
    for _ in range(3):  # both graph instances (the first was captured without the front)
        color.zero_()
        torch.cuda.synchronize()
        run.pipe.launch_graph([cam], stream=stream.cuda_stream)
        stream.synchronize()
        assert np.array_equal(color.cpu().numpy().view(np.uint32), ref["rgba"].view(np.uint32))
    run.close()


LIMIT = 1 << 16  # polls: the shortest limit that the front's barriers take, some 33 ms


def test_front_takes_set_limits_that_its_barriers_can_keep():
    scene, frame = case(seed=93)
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, "exact", capacity=int(o["state"][1]) + 256)
    for limit, front in ((0, True), (LIMIT, True), (LIMIT - 1, False), (2000, False)):
        run.pipe.set_wait_limit(limit)
        g = run.render(frame)
        assert (g["launches"] == 2) == front, limit
        assert_bit_exact(g, o)
    run.close()


@pytest.mark.parametrize("n", [200, 6000, 120001])  # one 256-splat unit, several, several per block
def test_front_barrier_expires_and_pipeline_recovers(n):
    import time
    import torch
    scene, frame = case(n, seed=94)
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, "exact", capacity=int(o["state"][1]) + 256)
    assert_bit_exact(run.render(frame), o)
    H, W = int(frame["height"]), int(frame["width"])
    color = torch.full((H, W, 4), 0.25, device="cuda")
    depth = torch.full((H, W), 0.5, device="cuda")
    torch.cuda.synchronize()
    run.pipe.set_wait_limit(LIMIT)
    run.pipe.debug_withhold_chunk()
    t0 = time.time()
    run.pipe.render(P.make_camera(frame), color.data_ptr(), depth.data_ptr(), 7, False, "rgba32f")
    with pytest.raises(P.GaussianPassError) as err:
        run.pipe.read_stats()
    assert time.time() - t0 < 30.0  # the kernel returned on its own
    assert err.value.status == P.abi.GS3D_ERROR_DEVICE_TIMEOUT
    assert "wait for other blocks expired" in str(err.value)
    assert run.pipe.last_launch_count() == 2
    assert (color == 0.25).all() and (depth == 0.5).all()
    # The hook applies to one render only; the next frames are complete and exact.
    for limit in (LIMIT, 0):
        run.pipe.set_wait_limit(limit)
        g = run.render(frame)
        assert g["launches"] == 2 and g["stats"]["deviceError"] == 0
        assert_bit_exact(g, o)
    run.close()
