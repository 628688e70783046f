"""The fused front of small launches where its cooperative launch is refused
and where its blocks wait in vain, made to happen without a GPU fault.

* A refused launch (an error code on the host, as on a stream that may use only
  a part of the device's SMs): the separate kernels render the frame. Nothing
  else may read the workspaces, which hold no frame yet.
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
