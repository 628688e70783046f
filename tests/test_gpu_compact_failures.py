"""gs3d_compact_visible_static after a call whose second kernel could not be
enqueued (an error on the host): the scratch of that call's compaction is left
as it was, and the calls after it still return the whole compaction."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [77, 300001])  # one chunk, and one per block of the grid
@pytest.mark.parametrize("captured", [False, True])
def test_a_refused_second_launch_spoils_no_later_call(n, captured):
    import torch
    P = pkg()
    lib = P.load()
    rng = np.random.Generator(np.random.PCG64(n))
    stream = torch.cuda.Stream()
    result = torch.zeros(2, dtype=torch.int32, device="cuda")
    out = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]

    def draw():
        vis = rng.random(n) < 0.4
        return vis, torch.from_numpy(np.where(vis, 7, -1).astype(np.int32)).cuda()

    def call(keys):
        return lib.gs3d_compact_visible_static(keys.data_ptr(), n, out[0].data_ptr(), out[1].data_ptr(),
                                               out[2].data_ptr(), result.data_ptr(), stream.cuda_stream)

    def check(vis):
        stream.synchronize()
        assert result.cpu().numpy().tolist() == [int(vis.sum()), 0]
        assert np.array_equal(out[0].cpu().numpy(), np.cumsum(vis) - vis)
        assert np.array_equal(out[2].cpu().numpy()[:vis.sum()], np.nonzero(vis)[0])
        for t in (*out, result):
            t.fill_(-1)
        torch.cuda.synchronize()

    vis, keys = draw()
    torch.cuda.synchronize()
    assert call(keys) == 0
    check(vis)
    lib.gs3d_debug_refuse_compact_finish()
    assert call(keys) == P.abi.GS3D_ERROR_CUDA
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    if captured:  # the first call after the refused one is captured, and runs after a direct one
        with torch.cuda.graph(graph, stream=stream):
            assert call(keys) == 0
    for _ in range(3):
        other, k = draw()
        torch.cuda.synchronize()
        assert call(k) == 0
        check(other)
        if captured:
            with torch.cuda.stream(stream):
                graph.replay()
            check(vis)
