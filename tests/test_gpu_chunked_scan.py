"""The chunked scans (visibility compaction, ordered-count scan): fewer visible
ranks than the grid was sized for, down to one unit of 256, and the static
entry point's scratch, which each call leaves ready for the next."""
import importlib

import numpy as np
import pytest

import oracle
from conftest import PKG_NAME, scenes
from gpu_harness import GpuRun, assert_bit_exact

pytestmark = pytest.mark.gpu

sc = scenes()
P = importlib.import_module(PKG_NAME)


@pytest.mark.parametrize("visible", [0, 1, 256, 257, 4097, 155648, 155649, 169000])
def test_visible_ranks_around_units_and_chunks(visible):
    # 170,001 ordinals fill the grid's 608 chunks (4 blocks of 152 SMs); the
    # visible ones lie anywhere among them, the others behind the camera.
    n = 170001
    scene = sc.uniform_cloud(n, seed=21, degree=0, log_scale=(-2.0, 0.1))
    scene["means"][:, :2] = scene["means"][:, :2] % 1.0
    frame = sc.make_frame(sc.look_at((0.5, 0.5, 30.0), (0.5, 0.5, 0.0)), 1000, 800, 20.0, 0.1, 100.0)
    shown = np.flatnonzero(oracle.render(scene, frame, 0)["tile_counts"])  # not too faint
    keep = np.random.Generator(np.random.PCG64(visible)).permutation(shown)[:visible]
    scene["means"][np.setdiff1d(np.arange(n), keep), 2] = 50.0
    o = oracle.render(scene, frame, 0)
    assert o["visible_state"][0] == visible
    run = GpuRun(scene, frame, "exact", capacity=max(int(o["state"][1]), 1))
    run.pipe.set_profiling(True)  # the separate kernels
    g = run.render(frame)
    run.close()
    assert g["launches"] > 2
    assert_bit_exact(g, o)


def test_static_scratch_is_ready_for_the_next_call():
    # Captured once and replayed, with calls of other sizes in between, and
    # with `result` at an address of no alignment.
    import torch
    lib = P.load()
    rng = np.random.Generator(np.random.PCG64(5))

    def case(n):
        vis = rng.random(n) < 0.4
        keys = torch.from_numpy(np.where(vis, 7, -1).astype(np.int32)).cuda()
        return keys, vis, [torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(3)]

    a, b = case(300001), case(77)
    result = torch.zeros(16, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()

    def call(c, at):
        keys, _, out = c
        assert lib.gs3d_compact_visible_static(keys.data_ptr(), len(keys), out[0].data_ptr(), out[1].data_ptr(),
                                               out[2].data_ptr(), result.data_ptr() + at, stream.cuda_stream) == 0

    def check(c, at):
        stream.synchronize()
        words = result.cpu().numpy()[at:at + 8].copy().view(np.uint32)
        assert words.tolist() == [int(c[1].sum()), 0]
        assert np.array_equal(c[2][2].cpu().numpy()[:words[0]], np.nonzero(c[1])[0])
        for t in c[2]:
            t.fill_(-1)
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    call(b, 0)
    check(b, 0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call(a, 4)
    for i in range(3):
        with torch.cuda.stream(stream):
            graph.replay()
        check(a, 4)
        call(b, 5 + i)
        check(b, 5 + i)
