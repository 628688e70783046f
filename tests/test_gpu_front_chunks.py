"""The fused front's chunked sort passes (front.cu: chunk_pass) against the
oracle: record counts at and around a tile of 2048 per block, where they begin,
with one or several tiles per block and a ragged last one."""
import numpy as np
import pytest

import oracle
from conftest import scenes
from gpu_harness import GpuRun, assert_bit_exact

pytestmark = pytest.mark.gpu

sc = scenes()


@pytest.mark.parametrize("digit_bits", [8, 4])  # one pass over the 64 tiles' ids, and two
@pytest.mark.parametrize("splats", ["limit", "limit + 1", "limit * 5 // 4", "limit * 7 // 2 + 11"])
def test_record_counts_around_the_chunked_passes(splats, digit_bits):
    import torch
    # A block per SM (few ordinals); every splat shown covers all 64 tiles.
    limit = torch.cuda.get_device_properties(0).multi_processor_count * 2048 // 64
    keep = eval(splats, {"limit": limit})
    n = 2 * keep
    assert n <= 256 * (limit // 32)
    scene = sc.uniform_cloud(n, seed=31, degree=0, log_scale=(1.7, 0.1))
    scene["means"][:, :3] *= 0.2
    frame = sc.make_frame(sc.look_at((0.0, 0.0, 11.0), (0, 0, 0)), 128, 128, 55.0, 0.1, 100.0)
    wide = np.flatnonzero(oracle.render(scene, frame, 0)["tile_counts"] == 64)
    assert len(wide) >= keep
    shown = np.zeros(n, bool)
    shown[wide[:keep]] = True
    scene["means"][~shown, 2] = 50.0  # behind the camera
    o = oracle.render(scene, frame, 0)
    assert o["visible_state"][0] == keep and o["state"][0] == 64 * keep
    run = GpuRun(scene, frame, "exact", capacity=64 * keep)
    run.pipe.set_tuning({"tile_digit_bits": digit_bits})
    g = run.render(frame)
    run.close()
    assert g["launches"] == 2
    assert_bit_exact(g, o)
