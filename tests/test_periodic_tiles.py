"""Tile boxes along a periodic axis (pass_exact.cu: periodic_tiles) and the
rasterizers' fixed image per patch (raster_impl.cuh: single_image).

The reference walks every tile of a periodic axis and tests those whose image
range is not empty (tileContribution.ts:84-114). The box must hold all of
these, each once and in ascending order; on the GPU every buffer of a periodic
frame equals the oracle's, from splats of a pixel to splats wider than the
period, where no box applies."""
import importlib

import numpy as np
import pytest

import oracle
from conftest import scenes

f32 = np.float32
sc = scenes()


def periodic_tiles(cen, r, period, tiles, ts):
    """The device function in numpy float32: the list of tiles walked."""
    inv = f32(1.0) / ts
    canon = cen - np.floor(cen / period) * period
    reach = r + f32(2.0) + f32(1e-6) * period
    if not (canon >= 0 and canon <= period and f32(2.0) * (reach + ts) < period):
        return list(range(tiles))
    last = tiles - 1
    a = max(int(np.floor((canon - reach) * inv)), 0)
    b = min(int(np.floor((canon + reach) * inv)), last)
    before, after = canon - period + reach, canon + period - reach
    if before >= 0:
        n0 = int(np.floor(before * inv)) + 1
        start, count, wrap = a - n0, n0 + tiles - a, n0
    elif after <= f32(tiles) * ts:
        f, n0 = min(int(np.floor(after * inv)), last), b + 1
        start, count, wrap = f - n0, n0 + tiles - f, n0
    else:
        start, count, wrap = a, b - a + 1, 0
    return [k if k < wrap else start + k for k in range(count)]


def image_tiles(cen, r, period, tiles, ts):
    """Tiles whose image range (boundary_tile_hit) is not empty."""
    canon = cen - np.floor(cen / period) * period
    t = np.arange(tiles).astype(f32) * ts
    first = np.ceil(((t - r) - canon) / period)
    last = np.floor((((t + ts) + r) - canon) / period)
    return set(np.nonzero(first <= last)[0].tolist())


@pytest.mark.parametrize("ts", [8, 16, 32])
@pytest.mark.parametrize("period", [1, 16, 17, 61, 97, 256, 1000, 2048, 3841, 40000])
def test_box_holds_every_tile_an_image_can_touch(period, ts):
    rng = np.random.Generator(np.random.PCG64(period * 64 + ts))
    tiles = -(-period // ts)
    p, t = f32(period), f32(ts)
    centres = np.concatenate([rng.uniform(-0.2, 1.2, 300) * period, rng.uniform(-5, 5, 60) * period,
                              rng.integers(0, tiles + 1, 60) * float(ts), [0.0, period, 1e9, -1e9, 3e7]])
    for cen in centres.astype(f32):
        r = f32(rng.integers(1, 12) if rng.random() < 0.7 else rng.integers(1, 334))
        with np.errstate(over="ignore", invalid="ignore"):
            walked = periodic_tiles(cen, r, p, tiles, t)
            need = image_tiles(cen, r, p, tiles, t)
        assert walked == sorted(set(walked)) and all(0 <= k < tiles for k in walked)
        assert need <= set(walked), (cen, r, period, ts)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["exact", "fp32", "half2"])
@pytest.mark.parametrize("axis,w,h,log_scale", [
    (1, 256, 64, (-3.5, 0.5)), (1, 333, 70, (-2.0, 1.2)), (1, 97, 64, (-0.5, 0.7)),
    (2, 64, 256, (-3.5, 0.5)), (2, 70, 333, (-2.0, 1.2)), (2, 64, 49, (-0.5, 0.7))])
def test_periodic_frames_equal_the_oracle(axis, w, h, log_scale, precision):
    from gpu_harness import FAST_COLOR_TOL, GpuRun, assert_bit_exact, psnr
    scene = sc.uniform_cloud(5000, seed=120 + axis, log_scale=log_scale)
    frame = sc.make_frame(sc.look_at((0.5, 1.0, 9.0), (0, 0, 0)), w, h, 75.0, 0.1, 100.0, boundary_axis=axis)
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, precision, capacity=max(int(o["state"][1]), 1))
    g = run.render(frame)
    run.close()
    if precision == "exact":
        assert_bit_exact(g, o)
        return
    assert_bit_exact(g, o, image=False, color_tol=FAST_COLOR_TOL)
    assert np.abs(g["rgba"] - o["rgba"]).max() <= (4e-3 if precision == "fp32" else 2e-2)  # the forms' tolerances
    assert psnr(g["rgba"][..., :3], o["rgba"][..., :3]) >= 50.0
