"""Box rows counted and emitted as one run of tiles (projection.cuh: row_span).

The device bounds the reference's tile test from both sides: tiles outside a
row's wide interval fail it, tiles of its narrow interval pass it, and only the
tiles between are tested. Checked here in float32 against the test itself
(tileContribution.ts:16-59) over random conics up to the condition number at
which the device falls back to walking the box; on the GPU every buffer of
frames full of wide boxes equals the oracle's."""
import importlib

import numpy as np
import pytest

import oracle
from conftest import scenes

f32 = np.float32
sc = scenes()


def tile_rect_test(cx, cy, k0, k1, k2, thr, tx, ty, ts):
    """The reference's test in float32, for arrays of tiles."""
    rminx, rminy = tx.astype(f32) * ts, f32(ty) * ts
    rmaxx, rmaxy = rminx + ts, rminy + ts
    x_left, x_right = cx < rminx, cx > rmaxx
    y_above, y_below = cy < rminy, cy > rmaxy
    in_x, in_y = ~(x_left | x_right), not (y_above or y_below)
    cornerx = np.where(x_left, rminx, rmaxx)
    cornery = rminy if y_above else rmaxy
    ex = np.where(x_left, ts, -ts)
    ey = ts if y_above else -ts
    dfx, dfy = cx - cornerx, cy - cornery
    txr = ((ex * k0) * dfx + (ex * k1) * dfy) / ((ex * k0) * ex)
    tyr = ((ey * k1) * dfx + (ey * k2) * dfy) / ((ey * k2) * ey)
    t_x = np.zeros_like(txr) if in_y else np.clip(txr, f32(0), f32(1))
    t_y = np.where(in_x, f32(0), np.clip(tyr, f32(0), f32(1)))
    dx, dy = (cornerx + t_x * ex) - cx, (cornery + t_y * ey) - cy
    sigma = f32(0.5) * ((k0 * dx) * dx + (k2 * dy) * dy) + (k1 * dx) * dy
    return (in_x & in_y) | (sigma <= thr)


def bounds(cx, cy, k0, k1, k2, thr, ty, x0, x1, extent, ts):
    """(a0, b0, a1, b1) of the device's row_span, or None where it gives the box up."""
    p = k1 * k1
    det = f32(float(k0) * float(k2) - float(p)) - f32(float(k1) * float(k1) - float(p))
    if not det > 0:
        return None
    delta = f32(1e-3) + f32(4e-6) * (k0 * k2 / det)
    if not (k0 > 0 and k2 > 0 and delta < f32(0.25)):
        return None
    m = f32(0.02) + f32(1e-6) * (abs(cx) + abs(cy) + extent)
    inv, ik0, slope, x2 = f32(1) / ts, f32(1) / k0, k1 / k2, k2 / det
    y0 = f32(ty) * ts - cy
    y1 = y0 + ts
    a0, b0, a1, b1 = 0, -1, 0, -1
    for wide in (True, False):
        grow = m if wide else -m
        level = (f32(2) * thr) * (f32(1) + delta if wide else f32(1) - delta)
        lo, hi, top = y0 - grow, y1 + grow, k0 * level
        near = min(max(f32(0), lo), hi)
        if not top >= det * near * near:
            break
        yr = slope * np.sqrt(level * x2)
        dr, dl = min(max(-yr, lo), hi), min(max(yr, lo), hi)
        xr = cx + (np.sqrt(max(top - det * dr * dr, f32(0))) - k1 * dr) * ik0 + grow
        xl = cx - (np.sqrt(max(top - det * dl * dl, f32(0))) + k1 * dl) * ik0 - grow
        if wide:
            a0, b0 = max(int(np.floor(xl * inv)), x0), min(int(np.floor(xr * inv)), x1)
        elif xl <= xr:
            a1, b1 = max(int(np.floor(xl * inv)), a0), min(int(np.floor(xr * inv)), b0)
    return a0, b0, a1, b1


def random_splat(rng, size):
    """Centre, conic and threshold of a projected splat on an image of `size` pixels."""
    s1, s2 = np.exp(rng.uniform(np.log(0.05), np.log(100.0), 2))
    th, var = rng.uniform(0, np.pi), rng.choice([0.3, 0.3, 0.05, 0.01])
    c, s = np.cos(th), np.sin(th)
    cov = np.array([[c * c * s1 * s1 + s * s * s2 * s2 + var, c * s * (s1 * s1 - s2 * s2)],
                    [0, s * s * s1 * s1 + c * c * s2 * s2 + var]])
    det = cov[0, 0] * cov[1, 1] - cov[0, 1] ** 2
    k0, k1, k2 = (f32(v) for v in (cov[1, 1] / det, -cov[0, 1] / det, cov[0, 0] / det))
    thr = f32(rng.choice([rng.uniform(0, 5.541), rng.uniform(0, 0.01), 5.5412636]))
    rx, ry = (f32(np.ceil(np.sqrt(2 * thr * cov[i, i]))) for i in (0, 1))
    cx, cy = f32(rng.uniform(-0.3, 1.3) * size), f32(rng.uniform(-0.3, 1.3) * size)
    if rng.random() < 0.1:  # on a tile corner
        cx, cy = f32(np.round(cx / 16) * 16), f32(np.round(cy / 16) * 16)
    return cx, cy, k0, k1, k2, thr, max(rx, f32(1)), max(ry, f32(1))


@pytest.mark.parametrize("ts,size", [(8, 700), (16, 1920), (16, 9000), (32, 4096)])
def test_bounds_hold_for_the_reference_test(ts, size):
    rng = np.random.Generator(np.random.PCG64(size + ts))
    t, tiles = f32(ts), -(-size // ts)
    rows = tested = given_up = 0
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        for _ in range(1200):
            cx, cy, k0, k1, k2, thr, rx, ry = random_splat(rng, size)
            x0, x1 = (int(np.clip(np.floor((cx + s * rx) / t), 0, tiles - 1)) for s in (-1, 1))
            y0, y1 = (int(np.clip(np.floor((cy + s * ry) / t), 0, tiles - 1)) for s in (-1, 1))
            cols = np.arange(x0, x1 + 1)
            for ty in range(y0, y1 + 1):
                got = bounds(cx, cy, k0, k1, k2, thr, ty, x0, x1, f32(2 * size), t)
                if got is None:
                    given_up += 1
                    break
                a0, b0, a1, b1 = got
                hits = tile_rect_test(cx, cy, k0, k1, k2, thr, cols, ty, t)
                assert not hits[(cols < a0) | (cols > b0)].any(), (cx, cy, k0, k1, k2, thr, ty)
                assert hits[(cols >= a1) & (cols <= b1)].all(), (cx, cy, k0, k1, k2, thr, ty)
                rows += 1
                tested += max(0, b0 - a0 + 1) - (b1 - a1 + 1 if a1 <= b1 else 0)
    assert rows > 2000 and tested < 0.25 * rows  # few tiles are left to the test


@pytest.mark.gpu
@pytest.mark.parametrize("log_scale,w,h,n", [
    ((-0.5, 0.8), 640, 400, 3000), ((0.8, 0.8), 641, 399, 1500), ((-1.5, 1.5), 333, 517, 8000),
    ((-2.0, 0.6), 1280, 720, 20000)])
def test_wide_boxes_equal_the_oracle(log_scale, w, h, n):
    # Near-degenerate axes among them: boxes the rows give up.
    from gpu_harness import GpuRun, assert_bit_exact
    scene = sc.clustered_cloud(n, seed=140 + w, clusters=8, centre_extent=4.0, std=(0.2, 1.5), log_scale=log_scale,
                               degenerate_fraction=0.1)
    frame = sc.make_frame(sc.look_at((0.5, 1.0, 12.0), (0, 0, 0)), w, h, 55.0, 0.1, 100.0, filter_variance=0.05)
    o = oracle.render(scene, frame, 0)
    run = GpuRun(scene, frame, "exact", capacity=max(int(o["state"][1]), 1))
    front = run.render(frame)
    run.pipe.set_profiling(True)
    separate = run.render(frame)
    run.close()
    assert_bit_exact(front, o)
    assert_bit_exact(separate, o)
