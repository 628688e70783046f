"""The benchmark's stage bytes follow the passes that the stages run (no GPU)."""
import importlib.util
import os

import pytest

from conftest import ROOT

spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
bench = importlib.util.module_from_spec(spec)
spec.loader.exec_module(bench)


@pytest.mark.parametrize("planes,passes", [
    ([(0.1, 1000.0)], 3),               # 27 bits
    ([(0.1, 100.0), (1.0, 1000.0)], 3), # the nearest near, the farthest far
    ([(1.0, 1.5)], 3),                  # 22 bits
    ([(1.0, 1.0 + 2.0 ** -9)], 2),      # 2^14 steps: 15 bits
    ([(1.0, 1.0 + 2.0 ** -16)], 1),
    ([(0.0, 1000.0)], 4),
    ([(0.001, 1000.0)], 4),             # a factor of a million: 28 bits
])
def test_depth_sort_passes_follow_the_planes(planes, passes):
    frames = [{"near": n, "far": f} for n, f in planes]
    assert bench.depth_sort_passes(frames) == passes
    per_pass = bench.stage_bytes("depth_sort", 10, 10, 0, 1, 1, 16, 1, 1, 8, False)
    assert bench.stage_bytes("depth_sort", 10, 10, 0, 1, 1, 16, passes, 1, 8, False) == passes * per_pass
