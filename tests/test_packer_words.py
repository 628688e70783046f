"""The packer's SH words at block edges and over the whole exponent range.

The device packer decides the shared exponent's rounding from the mantissa
alone (packer.cu: rounded_log2_ceil) and spreads a block's words over its
threads; both are checked against the C restatement, word for word."""
import importlib

import numpy as np
import pytest

import oracle
from conftest import PKG_NAME


def coefficients(n, C, seed):
    """Coefficient triples over the f32 exponent range, zeros and subnormals among them."""
    rng = np.random.Generator(np.random.PCG64(seed))
    e = rng.integers(-140, 127, (n, C - 1, 1)).astype(np.float64)
    v = (rng.uniform(-2.0, 2.0, (n, C - 1, 3)) * np.exp2(e)).astype(np.float32)
    v[rng.random((n, C - 1)) < 0.05] = 0.0
    return v


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1023])
@pytest.mark.parametrize("degree", [1, 2, 3])
def test_words_at_block_edges(n, degree):
    import torch
    P = importlib.import_module(PKG_NAME)
    C = (degree + 1) ** 2
    rng = np.random.Generator(np.random.PCG64(400 + n))
    centers = rng.uniform(-5, 5, (n, 3)).astype(np.float32)
    scales = np.full((n, 3), 0.25, np.float32)
    opacity = np.full(n, 0.5, np.float32)
    quats = np.tile(np.array([0, 0, 0, 1], np.float32), (n, 1))
    rgb = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    rest = coefficients(n, C, 500 + n + degree)
    o = oracle.pack_splats(centers, scales, opacity, quats, rgb, rest)
    t = [torch.from_numpy(a).cuda() for a in (centers, scales, opacity, quats, rgb, rest)]
    means = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
    shape = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    rot = torch.zeros(n, dtype=torch.int32, device="cuda")
    sh = torch.full((n * C + n,), 77, dtype=torch.int32, device="cuda")
    P.pack_splats(*t, 0, means, shape, rot, sh, n)
    torch.cuda.synchronize()
    got = sh.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[: n * C].reshape(n, C), o["sh"])
    assert (got[n * C:] == 77).all()  # the active-slot tail is the caller's
    assert np.array_equal(means.cpu().numpy().view(np.uint32), o["means"].view(np.uint32))
