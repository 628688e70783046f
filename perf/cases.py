"""Performance cases of the splatting pass: what a user of the framework has it do.

Single frames through ``TiledGaussianPipeline.render`` (the drop-in for the
reference's pass), batches of views through ``render_batch``, graph replays
(what the serving loop's lanes and a viewer's inner loop launch), the on-device
packer (streaming ingest) and the allocation-free visibility compaction.

Scenes are seeded on the GPU with the distributions of the benchmark
configurations (uniform cubes, anisotropic cluster mixtures, a far-origin
mixture with near-degenerate axes) and encoded here into the packed storage
buffers the pass consumes. ``exact`` renders the same packed bytes in float64
torch, without this repository's code.
"""
import importlib
import math

import numpy as np
import torch

P = importlib.import_module("3dgs_tile_webgpu_gb300")

SH_C0 = 0.28209479177387814
NEAR, FAR = 0.1, 1000.0
INVISIBLE = -1  # 0xffffffff as int32
FAR_ORIGIN = (1e5, 1e5, 0.0)
CONFIG3_SHARES = (50, 100, 250, 500, 750, 1000, 1500, 2000)  # eight clouds of uneven size


def _frame(name, splats, width, height, **kw):
    case = {"name": name, "kind": "frame", "scene": "uniform", "splats": splats, "width": width, "height": height,
            "degree": 3, "views": 1, "objects": 1, "precision": "fp32", "projection": "fp32", "sort": "float32",
            "antialias": "compensated", "boundary": "clip", "format": "rgba16f", "depth": False,
            "views_per_launch": 0}
    case.update(kw)
    return case


def listed():
    return [
        # A thumbnail or a first streamed-in LOD level: launches and latency are everything.
        _frame("frame_2k_160x90", 2048, 160, 90, degree=0, format="rgba32f", depth=True),
        # The plain single-cloud benchmark frame: 100k Gaussians at 720p, colour and depth as the pass node reads them.
        _frame("frame_100k_720p", 100_000, 1280, 720, depth=True),
        # The bit-exact form (regression images, reference comparisons) in an odd-sized window.
        _frame("exact_300k_1001x563", 300_000, 1001, 563, precision="exact", degree=2, format="rgba32f", depth=True),
        # A 360 degree panorama: periodic in x, 16-bit depth keys, classic anti-aliasing, a low SH degree.
        _frame("panorama_400k_2048x1024", 400_000, 2048, 1024, precision="half2", boundary="repeat-x",
               sort="packed16", antialias="classic", degree=1),
        # The large clustered benchmark scene as a viewer draws it: one FP32 view at a time at 1080p.
        _frame("frame_3m_1080p", 3_000_000, 1920, 1080, scene="clustered"),
        # The largest resident serving scene, one 1440p request in the half2 form.
        _frame("half2_6m_1440p", 6_000_000, 2560, 1440, precision="half2"),
        # A serving lane's small batch as a graph replay: four requests of mixed size on one mid-sized scene.
        _frame("graph_4x500k_mixed", 500_000, 1920, 1080, kind="graph", views=4, precision="half2"),
        # The headline throughput workload: 16 orbit cameras of the 3M scene at 1080p, 8 views per launch sequence.
        _frame("batch_16x3m_1080p", 3_000_000, 1920, 1080, kind="batch", scene="clustered", views=16,
               precision="half2", views_per_launch=8),
        # Many clouds, many views: eight objects with their own transforms, views of 480p to 4K in one batch.
        _frame("batch_8_objects_mixed", 1_500_000, 3840, 2160, kind="batch", views=8, objects=8),
        # Stress: far-origin scene in the FP64 projection form at 4K, hundreds of millions of intersections.
        _frame("far_12m_4k", 12_000_000, 3840, 2160, scene="far", precision="half2", projection="fp64"),
        # Streaming ingest: a decoded chunk of splats is encoded into the store's packed buffers.
        {"name": "pack_1m_sh3", "kind": "pack", "splats": 1_000_000, "degree": 3},
        # Visibility compaction for hosts that own all device memory.
        {"name": "compact_5m", "kind": "compact", "splats": 5_000_003, "visible": 0.72},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "frame", "graph", "batch", "batch", "far", "pack", "compact"))
    if kind == "pack":
        return {"kind": "pack", "splats": _log_int(rng, 5_000, 4_000_000), "degree": rng.randrange(4)}
    if kind == "compact":
        return {"kind": "compact", "splats": _log_int(rng, 1_000, 16_000_000), "visible": rng.uniform(0.05, 1.0)}
    width = _log_int(rng, 160, 3840)
    height = max(90, min(2160, int(width * rng.choice((0.5, 0.5625, 0.75, 1.0)))))
    if kind == "far":
        case = _frame("", _log_int(rng, 100_000, 8_000_000), width, height, scene="far", projection="fp64",
                      precision=rng.choice(("half2", "fp32")))
    else:
        case = _frame("", _log_int(rng, 2_000, 6_000_000), width, height, kind=kind,
                      scene=rng.choice(("uniform", "clustered")),
                      degree=rng.choice((0, 1, 2, 3, 3, 3)),
                      precision=rng.choice(("fp32", "fp32", "half2", "half2", "exact")),
                      sort=rng.choice(("float32", "float32", "float32", "packed16")),
                      antialias=rng.choice(("compensated", "compensated", "classic")),
                      boundary=rng.choice(("clip", "clip", "clip", "clip", "repeat-x", "repeat-y")),
                      format=rng.choice(("rgba16f", "rgba16f", "rgba32f")), depth=rng.random() < 0.4)
        if kind != "frame":
            case["views"] = rng.randrange(2, 13)
            case["splats"] = _log_int(rng, 2_000, 3_000_000)
            case["objects"] = rng.choice((1, 1, 8))
            if case["objects"] > 1:
                case["scene"] = "uniform"
            if kind == "batch":
                case["views_per_launch"] = rng.choice((0, 0, 4, 8))
        # Costs stay below the largest listed ones: a periodic axis tests every
        # tile along it, and the exact form is the slow one.
        most = 500_000 if case["boundary"] != "clip" else 8_000_000 if case["precision"] == "exact" else 24_000_000
        case["splats"] = min(case["splats"], most // case["views"])
    del case["name"]
    return case


# -- inputs -------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1000)
    return g


def _uniform(g, shape, lo, hi):
    return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=g)


def _normal(g, shape, mean, std):
    return torch.empty(shape, device="cuda").normal_(mean, std, generator=g)


def _clusters(g):
    return _uniform(g, (64, 3), -20.0, 20.0), _uniform(g, (64, 3), 0.2, 3.0)


def _linear(case, n, g, clusters):
    """Splat attributes: centres, natural-log scales, opacity, unit quaternions, DC colour."""
    clustered = case.get("scene", "uniform") != "uniform"
    if clustered:
        centre, std = clusters
        which = torch.randint(0, centre.shape[0], (n,), device="cuda", generator=g)
        means = centre[which] + _normal(g, (n, 3), 0.0, 1.0) * std[which]
    else:
        means = _uniform(g, (n, 3), -5.0, 5.0)
    far = case.get("scene") == "far"
    mu, sd = (-2.0, 1.0) if far else (-3.5, 0.7) if clustered else (-4.0, 0.5)
    log_scales = _normal(g, (n, 3), mu, sd)
    if far:
        means = means + torch.tensor(FAR_ORIGIN, device="cuda")
        flat = _uniform(g, (n,), 0.0, 1.0) < 0.05  # a near-degenerate axis
        axis = torch.randint(0, 3, (n, 1), device="cuda", generator=g)
        hit = torch.zeros((n, 3), dtype=torch.bool, device="cuda").scatter_(1, axis, flat[:, None])
        log_scales = torch.where(hit, torch.full_like(log_scales, -12.0), log_scales)
    opacity = torch.sigmoid(_normal(g, (n,), 0.5 if clustered else 0.0, 1.5))
    quats = _normal(g, (n, 4), 0.0, 1.0)
    quats = quats / quats.norm(dim=1, keepdim=True).clamp_min(1e-12)
    return means, log_scales, opacity, quats, _uniform(g, (n, 3), 0.0, 1.0)


def _f16_word(lo, hi):
    lo, hi = (x.to(torch.float16).view(torch.int16).to(torch.int32) & 0xFFFF for x in (lo, hi))
    return lo | (hi << 16)


def _oct101012(q):
    """Unit quaternions (n, 4) xyzw -> oct101012 words as int32."""
    q = torch.where(q[:, 3:] < 0, -q, q)
    theta = 2.0 * torch.arccos(q[:, 3].clamp(0.0, 1.0))
    s = torch.sin(theta * 0.5)
    axis = q[:, :3] / s[:, None].clamp_min(1e-12)
    axis = torch.where(s[:, None].abs() < 1e-6, torch.tensor([1.0, 0.0, 0.0], device=q.device), axis)
    p = axis[:, :2] / axis.abs().sum(1, keepdim=True)
    sign = torch.where(p >= 0, 1.0, -1.0)
    p = torch.where(axis[:, 2:] < 0, (1.0 - p.abs().flip(1)) * sign, p)
    uv = torch.floor(((p * 0.5 + 0.5) * 1023.0).clamp(0, 1023) + 0.5).to(torch.int32)
    r = torch.floor((theta / math.pi * 4095.0).clamp(0, 4095) + 0.5).to(torch.int32)
    return (r << 20) | (uv[:, 1] << 10) | uv[:, 0]


def _rgb8e8(c):
    """Signed RGB triples (..., 3) -> rgb8e8 words as int32."""
    top = c.abs().amax(-1)
    mantissa, e = torch.frexp(top)
    e = torch.where(mantissa == 0.5, e - 1, e).clamp(-126, 127)
    b = torch.floor(torch.ldexp(c, (7 - e)[..., None]) * (127.0 / 128.0) + 0.5).clamp(-127, 127).to(torch.int32) & 255
    word = b[..., 0] | (b[..., 1] << 8) | (b[..., 2] << 16) | ((e + 127) << 24)
    return torch.where(top > 0, word, torch.zeros_like(word))


def _scene(case, seed):
    """Packed buffers of one store, and how many splats each object holds."""
    n, degree = case["splats"], case["degree"]
    C = (degree + 1) ** 2
    g = _generator(seed)
    clusters = _clusters(g)
    means4 = torch.empty((n, 4), device="cuda")
    shape = torch.empty((n, 2), dtype=torch.int32, device="cuda")
    rot = torch.empty(n, dtype=torch.int32, device="cuda")
    sh = torch.empty(n * C + n, dtype=torch.int32, device="cuda")
    words = sh[: n * C].view(n, C)
    for a in range(0, n, 2_000_000):  # bounds the unpacked attributes' memory
        b = min(a + 2_000_000, n)
        means, ls, op, q, dc = _linear(case, b - a, g, clusters)
        means4[a:b, :3] = means
        shape[a:b, 0] = _f16_word(ls[:, 0], ls[:, 1])
        shape[a:b, 1] = _f16_word(ls[:, 2], op)
        rot[a:b] = _oct101012(q)
        words[a:b, 0] = _rgb8e8((dc - 0.5) / SH_C0)
        if C > 1:
            words[a:b, 1:] = _rgb8e8(_normal(g, (b - a, C - 1, 3), 0.0, 0.1))
    ids = torch.zeros(n, device="cuda")
    if case["objects"] > 1:
        edges = np.cumsum([0.0] + [float(s) for s in CONFIG3_SHARES[: case["objects"]]])
        edges = (edges / edges[-1] * n).astype(np.int64)
        for i in range(case["objects"]):
            ids[edges[i]:edges[i + 1]] = float(i)
    means4[:, 3] = ids
    sh[n * C:] = torch.arange(n, dtype=torch.int32, device="cuda")
    return {"n": n, "degree": degree, "means": means4, "shape": shape, "rot": rot, "sh": sh}


def _look_at(eye, target):
    z = eye - target
    z = z / np.linalg.norm(z)
    x = np.cross(np.array([0.0, 1.0, 0.0]), z)
    x = x / np.linalg.norm(x)
    m = np.eye(4)
    m[:3, 0], m[:3, 1], m[:3, 2], m[:3, 3] = x, np.cross(z, x), z, eye
    return m


def _projection(width, height, fov=60.0):
    top = NEAR * math.tan(math.radians(0.5 * fov))
    m = np.zeros((4, 4))
    m[0, 0], m[1, 1] = NEAR / (top * width / height), NEAR / top
    m[2, 2], m[2, 3], m[3, 2] = -(FAR + NEAR) / (FAR - NEAR), -2 * FAR * NEAR / (FAR - NEAR), -1.0
    return m


def _object_worlds(case, rng):
    if case["objects"] == 1:
        return [np.eye(4)]
    worlds = []
    for i in range(case["objects"]):  # rigid transforms with a uniform scale, on a ring
        q = rng.standard_normal(4)
        x, y, z, w = q / np.linalg.norm(q)
        m = np.eye(4)
        m[:3, :3] = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                              [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                              [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
        m[:3, :3] *= rng.uniform(0.5, 2.0)
        angle = 2 * math.pi * i / case["objects"]
        m[:3, 3] = (20.0 * math.cos(angle), rng.uniform(-3.0, 3.0), 20.0 * math.sin(angle))
        worlds.append(m)
    return worlds


def _frames(case, seed):
    """One frame description per view: seeded orbit cameras; the views of a batch differ in size."""
    rng = np.random.Generator(np.random.PCG64(int(seed) + 77))
    worlds = _object_worlds(case, rng)
    target = np.array(FAR_ORIGIN if case["scene"] == "far" else (0.0, 0.0, 0.0))
    radius = 45.0 if case["objects"] > 1 else 15.0 if case["scene"] == "uniform" else 30.0
    mixed = case["views"] > 1 and case["scene"] == "uniform"
    frames = []
    for i in range(case["views"]):
        width, height = case["width"], case["height"]
        if mixed:
            shrink = (1.0, 0.75, 0.5, 1 / 3)[i % 4]
            width, height = max(16, int(width * shrink)), max(16, int(height * shrink))
        az, el = 2 * math.pi * (i + rng.uniform()) / case["views"], math.radians(rng.uniform(-30.0, 30.0))
        eye = target + radius * np.array([math.cos(el) * math.sin(az), math.sin(el), math.cos(el) * math.cos(az)])
        camera = _look_at(eye, target)
        view = np.linalg.inv(camera)
        rows = np.zeros((len(worlds), 40))
        for k, world in enumerate(worlds):
            rows[k, :16] = world.T.reshape(-1)
            rows[k, 16:32] = (view @ world).T.reshape(-1)
            rows[k, 32:35] = (np.linalg.inv(world) @ np.append(eye, 1.0))[:3]
            rows[k, 35] = rows[k, 36] = 1.0
        frames.append({"projection": _projection(width, height).T.reshape(-1).astype(np.float32),
                       "view": view.T.reshape(-1).astype(np.float32), "width": width, "height": height,
                       "near": float(np.float32(NEAR)), "far": FAR, "objects": rows.astype(np.float32)})
    return frames


# -- the framework's calls ----------------------------------------------------

def _options(case):
    return {"raster_precision": case["precision"], "projection_precision": case["projection"],
            "depth_sort_mode": case["sort"], "antialias_mode": case["antialias"],
            "boundary_policy": case["boundary"], "intersection_capacity": max(262_144, 4 * case["splats"])}


def _grown(pipe, enqueue):
    """Renders until the intersection workspace holds the demand, with the capacity policy's headroom."""
    while True:
        enqueue()
        stats = pipe.read_stats()
        if not stats["overflow"]:
            return
        pipe.resize_intersections(int(stats["requestedIntersections"] * 1.25) + 256)


def _prepare_pack(case, seed):
    n, degree = case["splats"], case["degree"]
    C = (degree + 1) ** 2
    g = _generator(seed)
    means, ls, op, q, dc = _linear(case, n, g, _clusters(g))
    rest = _normal(g, (n, C - 1, 3), 0.0, 0.1) if C > 1 else None
    out = (torch.empty((n, 4), device="cuda"), torch.empty((n, 2), dtype=torch.int32, device="cuda"),
           torch.empty(n, dtype=torch.int32, device="cuda"),
           torch.zeros(n * C + n, dtype=torch.int32, device="cuda"))
    return {"kind": "pack", "source": (means.contiguous(), ls.exp(), op, q, dc, rest), "out": out, "n": n}


def _prepare_compact(case, seed):
    n = case["splats"]
    g = _generator(seed)
    keys = _uniform(g, (n,), NEAR, 60.0).view(torch.int32)
    keys = torch.where(_uniform(g, (n,), 0.0, 1.0) < case["visible"], keys, torch.full_like(keys, INVISIBLE))
    out = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]
    return {"kind": "compact", "lib": P.load(), "keys": keys, "n": n, "out": out,
            "result": torch.zeros(2, dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    if case["kind"] == "pack":
        return _prepare_pack(case, seed)
    if case["kind"] == "compact":
        return _prepare_compact(case, seed)
    scene, frames = _scene(case, seed), _frames(case, seed)
    data = P.gaussian_data_from_tensors(scene["n"], scene["n"], scene["degree"], scene["means"], scene["shape"],
                                        scene["rot"], scene["sh"])
    pipe = P.TiledGaussianPipeline(data, _options(case))
    cams = [P.make_camera(f) for f in frames]
    dtype = torch.float16 if case["format"] == "rgba16f" else torch.float32
    color = [torch.zeros((f["height"], f["width"], 4), dtype=dtype, device="cuda") for f in frames]
    depth = [torch.zeros((f["height"], f["width"]), device="cuda") if case["depth"] else None for f in frames]
    state = {"kind": case["kind"], "scene": scene, "data": data, "pipe": pipe, "cams": cams, "color": color,
             "depth": depth, "format": case["format"]}
    state["views"] = [(data, cam, f["width"], f["height"], c.data_ptr(), d.data_ptr() if d is not None else 0,
                       case["format"]) for cam, f, c, d in zip(cams, frames, color, depth)]
    torch.cuda.current_stream().synchronize()  # the pass reads the buffers from its own stream
    if case["kind"] == "frame":
        pipe.prepare_frame(frames[0]["width"], frames[0]["height"])
        _grown(pipe, lambda: run(state))
        return state
    if case["views_per_launch"]:
        pipe.set_tuning({"views_per_launch": case["views_per_launch"]})
    _grown(pipe, lambda: pipe.render_batch(state["views"]))
    if case["kind"] == "graph":
        state["stream"] = torch.cuda.Stream()
        pipe.capture_graph(state["views"], state["stream"].cuda_stream)
    return state


def run(state):
    kind = state["kind"]
    if kind == "pack":
        means, shape, rot, sh = state["out"]
        P.pack_splats(*state["source"], 0, means, shape, rot, sh, state["n"])
        return list(state["out"])
    if kind == "compact":
        off, keys, ids = state["out"]
        P._raise(state["lib"], state["lib"].gs3d_compact_visible_static(
            state["keys"].data_ptr(), state["n"], off.data_ptr(), keys.data_ptr(), ids.data_ptr(),
            state["result"].data_ptr(), 0))
        return {"offsets": off, "keys": keys, "ids": ids, "result": state["result"]}
    pipe = state["pipe"]
    if kind == "frame":
        depth = state["depth"][0]
        pipe.render(state["cams"][0], state["color"][0].data_ptr(), depth.data_ptr() if depth is not None else 0,
                    color_format=state["format"])
    elif kind == "batch":
        pipe.render_batch(state["views"])
    else:
        pipe.launch_graph(state["cams"], stream=state["stream"].cuda_stream)
    return {"color": state["color"], "depth": state["depth"]}


# -- what a pass cannot do without --------------------------------------------

def work(case):
    n = case["splats"]
    if case["kind"] == "compact":
        return {"bytes": 4.0 * n + 4.0 * n + 8.0 * n * case["visible"], "flops": 0.0}
    C = (case["degree"] + 1) ** 2
    if case["kind"] == "pack":
        return {"bytes": n * (4.0 * (14 + 3 * (C - 1)) + 28.0 + 4.0 * C), "flops": n * (60.0 + 15.0 * C)}
    pixels = sum(f["width"] * f["height"] for f in _frames(case, 0))
    out = (8 if case["format"] == "rgba16f" else 16) + (4 if case["depth"] else 0)
    # Each splat's projection takes some 400 operations and its colour 10 per
    # coefficient; a pixel blends some tens of samples at about 22 each.
    return {"bytes": n * (32.0 + 4.0 * C) + float(pixels * out),
            "flops": case["views"] * n * (400.0 + 10.0 * C) + pixels * 50.0 * 22.0}


# -- the same images in float64 -----------------------------------------------

def _decode(scene):
    """Packed words -> float64 centres, object ids, scales, opacity, quaternions, SH coefficients."""
    n, C = scene["n"], (scene["degree"] + 1) ** 2
    half = scene["shape"].view(torch.float16).view(n, 4).double()
    p = scene["rot"].to(torch.int64) & 0xFFFFFFFF
    px, py = (((p >> s) & 1023).double() / 1023.0 * 2.0 - 1.0 for s in (0, 10))
    z = 1.0 - px.abs() - py.abs()
    t = (-z).clamp_min(0.0)
    axis = torch.stack([torch.where(px >= 0, px - t, px + t), torch.where(py >= 0, py - t, py + t), z], 1)
    axis = axis / axis.norm(dim=1, keepdim=True)
    half_angle = (p >> 20).double() / 4095.0 * (math.pi / 2)
    quat = torch.cat([axis * half_angle.sin()[:, None], half_angle.cos()[:, None]], 1)
    means = scene["means"].double()
    return means[:, :3], means[:, 3].long(), half[:, :3].exp(), half[:, 3], quat, scene["sh"][: n * C].view(n, C)


def _sh_colour(words, degree, d):
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    basis = [torch.full_like(x, SH_C0)]
    if degree >= 1:
        basis += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree >= 2:
        xx, yy, zz = x * x, y * y, z * z
        basis += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
                  -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy)]
    if degree >= 3:
        basis += [-0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
                  -0.4570457994644658 * y * (4 * zz - xx - yy),
                  0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
                  -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
                  -0.5900435899266435 * x * (xx - 3 * yy)]
    colour = torch.full((x.numel(), 3), 0.5, dtype=torch.float64, device=x.device)
    for k, w in enumerate(basis):
        word = words[:, k].to(torch.int64) & 0xFFFFFFFF
        scale = torch.exp2(((word >> 24) & 255).double() - 127.0)
        for c in range(3):
            byte = (word >> (8 * c)) & 255
            signed = torch.where(byte > 127, byte - 256, byte).double()
            colour[:, c] += w * scale * (signed / 127.0).clamp_min(-1.0)
    return colour.clamp(0.0, 1.0)


def _exact_projection(decoded, degree, frame, case):
    """Visible splats of one view, front to back: centre, conic, opacity, extents, depth, colour."""
    pos, obj, scale, opacity, q, words = decoded
    rows = torch.from_numpy(frame["objects"]).to(pos.device).double()
    proj = torch.from_numpy(frame["projection"]).to(pos.device).double().view(4, 4).T
    mv = rows[:, 16:32].view(-1, 4, 4).transpose(1, 2)[obj]
    W, H = float(frame["width"]), float(frame["height"])
    view = (mv[:, :3, :3] * pos[:, None, :]).sum(2) + mv[:, :3, 3]
    depth = -view[:, 2]
    keep = (depth > frame["near"]) & (depth < frame["far"])
    x, y, z, w = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
    M = torch.bmm(mv[:, :3, :3], R) * scale.clamp_min(1e-7)[:, None, :]
    hom = torch.cat([view, torch.ones_like(depth)[:, None]], 1) @ proj.T
    cx, cy = (hom[:, 0] / hom[:, 3] * 0.5 + 0.5) * W, (0.5 - hom[:, 1] / hom[:, 3] * 0.5) * H
    fx, fy = 0.5 * W * proj[0, 0], 0.5 * H * proj[1, 1]
    zero = torch.zeros_like(depth)
    a0 = (torch.stack([fx / depth, zero, fx * view[:, 0] / depth ** 2], 1)[:, None, :] @ M)[:, 0]
    a1 = (torch.stack([zero, -fy / depth, -fy * view[:, 1] / depth ** 2], 1)[:, None, :] @ M)[:, 0]
    c00, c01, c11 = (a0 * a0).sum(1), (a0 * a1).sum(1), (a1 * a1).sum(1)
    det0 = (c00 * c11 - c01 * c01).clamp_min(0.0)
    s00, s01, s11 = c00 + 0.3, c01, c11 + 0.3
    mid, rad = 0.5 * (s00 + s11), (0.25 * (s00 - s11) ** 2 + s01 * s01).sqrt()
    lo, hi = (mid - rad).clamp(1e-6, 1e4), (mid + rad).clamp(1e-6, 1e4)
    th = 0.5 * torch.atan2(2 * s01, s00 - s11)
    cs, sn = th.cos(), th.sin()
    s00, s01, s11 = lo * sn * sn + hi * cs * cs, (hi - lo) * cs * sn, lo * cs * cs + hi * sn * sn
    det = s00 * s11 - s01 * s01
    keep &= (hom[:, 3] > 0) & (det > 1e-8) & (s00 <= 1e4) & (s11 <= 1e4)
    op = opacity.clamp(0.0, 1.0)
    if case["antialias"] == "compensated":
        op = op * (det0 / det).clamp(0.0, 1.0).sqrt()
    keep &= op >= 1.0 / 255.0
    keep &= rows[obj, 36] > 0
    i = keep.nonzero()[:, 0]
    key = depth[i]
    if case["sort"] == "packed16":
        key = torch.round(((key - frame["near"]) / (frame["far"] - frame["near"])).clamp(0, 1) * 65535.0)
    i = i[torch.sort(key, stable=True)[1]]
    thr = (op[i] * 255.0).log()
    direction = pos[i] - rows[obj[i], 32:35]
    colour = _sh_colour(words[i], degree, direction / direction.norm(dim=1, keepdim=True))
    return {"cx": cx[i], "cy": cy[i], "a": (s11 / det)[i], "b": (-s01 / det)[i], "c": (s00 / det)[i], "op": op[i],
            "ex": (2 * thr * s00[i]).sqrt().ceil(), "ey": (2 * thr * s11[i]).sqrt().ceil(), "depth": depth[i],
            "rgb": colour}


def _exact_image(s, frame, case):
    """Front-to-back blend of every (pixel, splat) pair, band by band of pixel rows."""
    W, H = frame["width"], frame["height"]
    dev = s["cx"].device
    wrap = {"clip": 0, "repeat-x": 1, "repeat-y": 2}[case["boundary"]]
    acc = torch.zeros((H * W, 5), dtype=torch.float64, device=dev)  # rgb, depth, log transmittance
    x0, x1 = torch.floor(s["cx"] - s["ex"]).long(), torch.ceil(s["cx"] + s["ex"]).long()
    y0, y1 = torch.floor(s["cy"] - s["ey"]).long(), torch.ceil(s["cy"] + s["ey"]).long()
    if wrap == 1:
        x1 = torch.minimum(x1, x0 + W)
    else:
        x0, x1 = x0.clamp(0, W), x1.clamp(0, W)
    if wrap == 2:
        y1 = torch.minimum(y1, y0 + H)
    else:
        y0, y1 = y0.clamp(0, H), y1.clamp(0, H)
    area = (x1 - x0).clamp_min(0) * (y1 - y0).clamp_min(0)
    bands = max(1, min(H, int(float(area.sum()) / 3e7) + 1))
    bands = bands if wrap == 0 else 1 if float(area.sum()) < 2e8 else None
    if bands is None:
        return None
    for k in range(bands):
        r0, r1 = H * k // bands, H * (k + 1) // bands
        ya, yb = (y0, y1) if wrap == 2 else (y0.clamp(r0, r1), y1.clamp(r0, r1))
        w, h = (x1 - x0).clamp_min(0), (yb - ya).clamp_min(0)
        i = ((w > 0) & (h > 0)).nonzero()[:, 0]
        if not i.numel():
            continue
        count = w[i] * h[i]
        rep = torch.repeat_interleave(i, count)
        at = torch.arange(rep.numel(), device=dev) - torch.repeat_interleave(count.cumsum(0) - count, count)
        px, py = x0[rep] + at % w[rep], ya[rep] + torch.div(at, w[rep], rounding_mode="floor")
        if wrap == 1:
            px = px % W
        if wrap == 2:
            py = py % H
        dx, dy = px.double() + 0.5 - s["cx"][rep], py.double() + 0.5 - s["cy"][rep]
        a, b, c = s["a"][rep], s["b"][rep], s["c"][rep]
        if wrap == 1:
            dx = dx - torch.floor((dx + b * dy / a) / W + 0.5) * W
        if wrap == 2:
            dy = dy - torch.floor((dy + b * dx / c) / H + 0.5) * H
        alpha = (s["op"][rep] * torch.exp(-0.5 * (a * dx * dx + 2 * b * dx * dy + c * dy * dy))).clamp_max(0.99)
        use = (alpha >= 1.0 / 255.0).nonzero()[:, 0]
        pixel, order = torch.sort((py[use] * W + px[use]), stable=True)
        use = use[order]
        if not use.numel():
            continue
        alpha, rep = alpha[use], rep[use]
        logs = torch.log1p(-alpha)
        before = logs.cumsum(0) - logs
        first = torch.ones_like(pixel, dtype=torch.bool)
        first[1:] = pixel[1:] != pixel[:-1]
        start = before[first][first.long().cumsum(0) - 1]
        trans = torch.exp(before - start)
        live = trans >= 1e-4  # a pixel stops once its transmittance is below the threshold
        contrib = torch.where(live, trans * alpha, torch.zeros_like(alpha))
        add = torch.cat([s["rgb"][rep] * contrib[:, None], (s["depth"][rep] * contrib)[:, None],
                         torch.where(live, logs, torch.zeros_like(logs))[:, None]], 1)
        acc.index_add_(0, pixel, add)
    t = acc[:, 4].exp()
    colour = torch.cat([acc[:, :3], (1.0 - t)[:, None]], 1).view(H, W, 4)
    if not case["depth"]:
        return colour, None
    cover = 1.0 - t
    z = acc[:, 3] / cover.clamp_min(1e-300)
    near, far = frame["near"], frame["far"]
    device_depth = ((near - z) * far / ((far - near) * -z.clamp_min(1e-300))).clamp(0.0, 1.0)
    depth = torch.where((cover > 0.95) & (z > 0), device_depth, torch.ones_like(z))
    return colour, depth.view(H, W)


def exact(case, seed):
    """The images in float64 (all but the packer's centres, and the compaction's outputs, are whole numbers)."""
    if case["kind"] == "pack":
        g = _generator(seed)
        centres = _linear(case, case["splats"], g, _clusters(g))[0].double()
        return [torch.cat([centres, torch.zeros_like(centres[:, :1])], 1), None, None, None]
    if case["kind"] == "compact" or case["scene"] == "far":
        return None
    if case["precision"] == "exact" and case["splats"] > 1_000_000:
        return None
    scene, frames = _scene(case, seed), _frames(case, seed)
    decoded = _decode(scene)
    colour, depth = [], []
    for k, frame in enumerate(frames):
        image = None
        if k < 4:  # the first views of a batch; all of them would take too long
            image = _exact_image(_exact_projection(decoded, scene["degree"], frame, case), frame, case)
        colour.append(None if image is None else image[0])
        depth.append(None if image is None else image[1])
    return {"color": colour, "depth": depth}
