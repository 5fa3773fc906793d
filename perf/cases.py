"""The workloads this framework's speed is judged by: what a user has it do, through
``rasterization()``, ``lidar_rasterization()`` and the lidar point preparation ops.

Sizes, sensors and value distributions are those of the benchmark configurations
(``splatad_b200/scenes.py``), from the smallest to the largest of them, plus odd and ragged sizes in
between. Every input is drawn on the GPU from the seed alone; the seed also turns the sensors, so
that another seed is another scene seen from another direction.

A case is a dict: ``kind`` ("lidar", "camera" or "points"), the sizes, and the options. ``train``
adds the backward pass: the cotangents of the images are given (what a loss hands back), gradients
come back on the parameters and, as a densification strategy reads them, on ``meta["means2d"]``.
"""

import math

import torch

import splatad_b200
from splatad_b200 import ops, scenes

TILE_WIDTH, TILE_HEIGHT = 32, 8   # lidar tiles of every configuration
TILE_SIZE = 16                    # camera tiles


def listed():
    return [
        # A small scan: the configuration the CPU oracle can follow end to end (32 x 512 points). Host
        # work and launches count.
        dict(name="lidar_small", kind="lidar", n=20_000, sensors=1, beams=32, columns=512, features=4,
             rolling=False, moving=False, antialiased=False, train=False),
        # The same as a training step.
        dict(name="lidar_small_train", kind="lidar", n=20_000, sensors=1, beams=32, columns=512, features=4,
             rolling=False, moving=False, antialiased=False, train=True),
        # A ragged scan in training: 64 beams, a column count that fills no tile, an odd feature count,
        # moving Gaussians (dynamic actors), opacities compensated for the blur.
        dict(name="lidar_odd_train", kind="lidar", n=173_281, sensors=1, beams=64, columns=1083, features=7,
             rolling=True, moving=True, antialiased=True, train=True),
        # The headline frame: a million Gaussians, a 128 x 1800 rolling-shutter sweep, 16 features.
        dict(name="lidar_frame", kind="lidar", n=1_000_000, sensors=1, beams=128, columns=1800, features=16,
             rolling=True, moving=False, antialiased=False, train=False),
        # The same frame as a training step.
        dict(name="lidar_train", kind="lidar", n=1_000_000, sensors=1, beams=128, columns=1800, features=16,
             rolling=True, moving=False, antialiased=False, train=True),
        # A preview image: few Gaussians with plain colours, small image, [C, N] layout.
        dict(name="camera_small", kind="camera", n=30_000, sensors=1, width=640, height=360, channels=3, sh=-1,
             packed=False, mode="RGB", moving=False, antialiased=False, absgrad=False, train=False),
        # The camera benchmark frame: 500 k Gaussians, SH degree 3, packed, colour and depth.
        dict(name="camera_frame", kind="camera", n=500_000, sensors=1, width=1920, height=1080, channels=3, sh=3,
             packed=True, mode="RGB+D", moving=True, antialiased=False, absgrad=False, train=False),
        # The same frame as a training step.
        dict(name="camera_train", kind="camera", n=500_000, sensors=1, width=1920, height=1080, channels=3, sh=3,
             packed=True, mode="RGB+D", moving=True, antialiased=False, absgrad=False, train=True),
        # Feature splatting in training: 13 feature channels and the expected depth, a ragged image, [C, N]
        # layout, antialiased opacities, absolute gradients for the densification.
        dict(name="camera_odd_train", kind="camera", n=211_003, sensors=1, width=1237, height=719, channels=13, sh=-1,
             packed=False, mode="RGB+ED", moving=True, antialiased=True, absgrad=True, train=True),
        # Three cameras of a rig in one training step.
        dict(name="rig_train", kind="camera", n=400_000, sensors=3, width=1280, height=720, channels=3, sh=3,
             packed=True, mode="RGB+D", moving=False, antialiased=False, absgrad=False, train=True),
        # The whole rig: six 1920 x 1080 cameras looking at two million Gaussians in one packed call.
        dict(name="rig_frame", kind="camera", n=2_000_000, sensors=6, width=1920, height=1080, channels=3, sh=3,
             packed=True, mode="RGB+D", moving=False, antialiased=False, absgrad=False, train=False),
        # A recorded sweep of 128 x 1800 returns brought into the raster image the lidar render takes.
        dict(name="points_image", kind="points", n=230_400, sensors=1, beams=128, columns=1800),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("lidar", "lidar", "camera", "camera", "rig", "points"))
    if kind == "points":
        beams, columns = rng.randint(32, 128), rng.randint(512, 1800)
        return dict(kind="points", n=_spread(rng, 10_000, 460_800), sensors=rng.choice((1, 1, 2)), beams=beams,
                    columns=columns)
    if kind == "lidar":
        return dict(kind="lidar", n=_spread(rng, 20_000, 1_000_000), sensors=rng.choice((1, 1, 1, 2)),
                    beams=rng.randint(32, 128), columns=rng.randint(512, 1800), features=rng.randint(1, 20),
                    rolling=rng.random() < 0.8, moving=rng.random() < 0.4, antialiased=rng.random() < 0.2,
                    train=rng.random() < 0.5)
    rig = kind == "rig"
    sh = rng.choice((3, 3, 2, -1))
    return dict(kind="camera", n=_spread(rng, 30_000, 1_000_000 if rig else 500_000),
                sensors=rng.randint(2, 6) if rig else 1, width=_spread(rng, 640, 1920), height=_spread(rng, 360, 1080),
                channels=3 if sh >= 0 else rng.choice((3, 3, 8, 13)), sh=sh, packed=rng.random() < 0.6,
                mode=rng.choice(("RGB", "RGB+D", "RGB+ED")), moving=rng.random() < 0.5,
                antialiased=rng.random() < 0.3, absgrad=rng.random() < 0.3,
                train=rng.random() < (0.3 if rig else 0.5))


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
def _gaussians(case, n, g, device):
    """Means, quaternions, scales and opacities of the benchmark scenes: the box around a lidar or a
    rig, or the box in front of a single camera."""
    def uniform(lo, hi):
        return torch.rand(n, generator=g, device=device) * (hi - lo) + lo

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=device)

    if case["kind"] == "camera" and case["sensors"] == 1:
        means = torch.stack([uniform(-50, 50), uniform(-5, 5), uniform(0.5, 100.5)], -1)
        scales = torch.exp(normal(n, 3) * 0.7 - 1.5)
    else:
        means = torch.stack([uniform(-40, 40), uniform(-40, 40), uniform(-2, 4)], -1)
        scales = torch.exp(normal(n, 3) * 0.5 - 1.0)
    quats = torch.nn.functional.normalize(normal(n, 4), dim=-1)
    opacities = torch.sigmoid(normal(n))
    return means, quats, scales, opacities


def _velocities(n, g, device):
    """One Gaussian in ten moves, with N(0, 2) m/s per axis."""
    v = torch.randn(n, 3, generator=g, device=device) * 2.0
    return v * (torch.rand(n, 1, generator=g, device=device) < 0.1)


def _beams(count):
    return scenes.beams_128() if count == 128 else torch.linspace(-25.0, 15.0, count)


def _yaw(degrees):
    c, s = math.cos(math.radians(degrees)), math.sin(math.radians(degrees))
    m = torch.eye(4)
    m[:2, :2] = torch.tensor([[c, s], [-s, c]])
    return m


def _lidar(case, g, device, turn):
    C, W = case["sensors"], case["columns"]
    elev = _beams(case["beams"])
    H = elev.numel()
    pts = torch.empty(C, H, W, 4, device=device)
    pts[..., 0] = -180.0 + (torch.arange(W, device=device) + 0.5) * (360.0 / W)
    pts[..., 1] = elev.to(device)[:, None]
    pts[..., 2] = torch.rand(C, H, W, generator=g, device=device) * 78 + 2
    pts[..., 3] = torch.linspace(-0.05, 0.05, W, device=device) if case["rolling"] else 0.0
    viewmats = torch.stack([_yaw(turn) for _ in range(C)])
    viewmats[:, 0, 3] = -torch.arange(C, dtype=torch.float32)   # sensors a metre apart
    kw = dict(viewmats=viewmats.to(device), raster_pts=pts,
              tile_elevation_boundaries=scenes.elevation_boundaries(elev, TILE_HEIGHT).to(device),
              min_azimuth=-180.0, max_azimuth=180.0, min_elevation=float(elev[0]) - 1.0,
              max_elevation=float(elev[-1]) + 1.0, n_elevation_channels=H, azimuth_resolution=360.0 / W,
              tile_width=TILE_WIDTH, tile_height=TILE_HEIGHT,
              rasterize_mode="antialiased" if case["antialiased"] else "classic")
    if case["rolling"]:
        kw.update(linear_velocity=torch.tensor([[15.0, 0.0, 0.0]], device=device).repeat(C, 1),
                  angular_velocity=torch.tensor([[0.0, 0.0, 0.1]], device=device).repeat(C, 1),
                  rolling_shutter_time=torch.full((C,), 0.1, device=device))
    return kw


def _cameras(case, device, turn):
    C, W, H = case["sensors"], case["width"], case["height"]
    if C == 1:
        # in front of the box it was drawn for, looking up to a few degrees aside
        viewmats = torch.eye(4)[None].clone()
        c, s = math.cos(math.radians(turn)), math.sin(math.radians(turn))
        viewmats[0, 0, 0], viewmats[0, 0, 2], viewmats[0, 2, 0], viewmats[0, 2, 2] = c, -s, s, c
    else:
        viewmats = scenes.yawed_camera_viewmats([turn + i * 360.0 / C for i in range(C)])
    Ks = torch.tensor([[0.625 * W, 0.0, 0.5 * W], [0.0, 0.625 * W, 0.5 * H], [0.0, 0.0, 1.0]])[None].repeat(C, 1, 1)
    return dict(viewmats=viewmats.to(device), Ks=Ks.to(device), width=W, height=H,
                linear_velocity=torch.tensor([[10.0, 0.0, 0.0]], device=device).repeat(C, 1),
                angular_velocity=torch.zeros(C, 3, device=device),
                rolling_shutter_time=torch.full((C,), 0.03, device=device), tile_size=TILE_SIZE,
                sh_degree=case["sh"] if case["sh"] >= 0 else None, packed=case["packed"], render_mode=case["mode"],
                rasterize_mode="antialiased" if case["antialiased"] else "classic", absgrad=case["absgrad"])


def _channels(case):
    """Rendered channels."""
    if case["kind"] == "lidar":
        return case["features"] + 1
    return case["channels"] + (1 if case["mode"] != "RGB" else 0)


def _colour_shape(case, n):
    """Per-Gaussian colour or feature values of a case."""
    if case["kind"] == "lidar":
        return (case["sensors"], n, case["features"])
    return (n, (case["sh"] + 1) ** 2, 3) if case["sh"] >= 0 else (n, case["channels"])


def prepare(case, seed):
    device = "cuda"
    g = torch.Generator(device=device).manual_seed(seed)
    n, C = case["n"], case["sensors"]
    if case["kind"] == "points":
        # returns of a sweep: azimuths over the turn, elevations around the beams, range, two attributes
        elev = _beams(case["beams"])
        lo, hi = float(elev[0]), float(elev[-1])
        pts = torch.rand(C, n, 5, generator=g, device=device)
        pts[..., 0] = pts[..., 0] * 360.0 - 180.0
        pts[..., 1] = pts[..., 1] * (hi - lo) + lo
        pts[..., 2] = pts[..., 2] * 78.0 + 2.0
        bounds = scenes.elevation_boundaries(elev, TILE_HEIGHT).to(device)
        return dict(case=case, points=pts, bounds=bounds)
    means, quats, scales, opacities = _gaussians(case, n, g, device)
    colours = torch.randn(_colour_shape(case, n), generator=g, device=device)
    if case["kind"] == "camera":
        colours = colours * 0.3 if case["sh"] >= 0 else torch.sigmoid(colours)
    params = dict(means=means, quats=quats, scales=scales, opacities=opacities)
    params["lidar_features" if case["kind"] == "lidar" else "colors"] = colours
    velocities = _velocities(n, g, device) if case["moving"] else None
    turn = (seed * 37) % 360
    if case["kind"] == "lidar":
        sensor = _lidar(case, g, device, turn)
        shape = (C, case["beams"], case["columns"])
    else:
        sensor = _cameras(case, device, turn if C > 1 else (turn % 9) - 4)
        shape = (C, case["height"], case["width"])
    state = dict(case=case, params=params, velocities=velocities, sensor=sensor)
    if case["train"]:
        for p in params.values():
            p.requires_grad_(True)
        # cotangents of a mean over the image: features, alphas and, for a lidar, the alpha sum
        widths = (_channels(case), 1) + ((1,) if case["kind"] == "lidar" else ())
        state["cotangents"] = [torch.randn(shape + (w,), generator=g, device=device) / math.prod(shape)
                               for w in widths]
    return state


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------
# What comes back of ``meta``: everything whose length the sizes of the case decide. The lists and packed
# rows are as long as the scene makes them; they are made all the same, and the tile offsets (where every
# list begins), the images and the gradients are made from them.
_META = ("isect_offsets", "median_depths")
_META_UNPACKED = ("radii", "means2d", "depths", "conics", "tiles_per_gauss")


def run(state):
    case = state["case"]
    if case["kind"] == "points":
        tile_azimuth = 360.0 / case["columns"] * TILE_WIDTH
        grid_w, grid_h = math.ceil(360.0 / tile_azimuth), math.ceil(case["beams"] / TILE_HEIGHT)
        points = state["points"]
        ids, flat = ops.map_points_to_lidar_tiles(points[..., :2], state["bounds"], tile_azimuth, -180.0)
        offsets = ops.points_mapping_offset_encode(ids, case["sensors"], grid_w, grid_h)
        image = ops.populate_image_from_points(points, case["columns"], case["beams"], TILE_WIDTH, TILE_HEIGHT,
                                               offsets, flat)
        return dict(ids=ids, flat=flat, offsets=offsets, image=image)
    params = state["params"]
    for p in params.values():
        p.grad = None
    render = splatad_b200.lidar_rasterization if case["kind"] == "lidar" else splatad_b200.rasterization
    *images, meta = render(velocities=state["velocities"], **params, **state["sensor"])
    packed = case.get("packed", False)
    out = dict(images=images, meta={k: meta[k] for k in _META + (() if packed else _META_UNPACKED) if k in meta})
    if case["train"]:
        meta["means2d"].retain_grad()
        torch.autograd.backward(images, state["cotangents"])
        out["grads"] = {k: p.grad for k, p in params.items()}
        if not packed:
            out["means2d_grad"] = meta["means2d"].absgrad if case.get("absgrad") else meta["means2d"].grad
    return out


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _estimate(case):
    """(visible share of the Gaussians, list entries) per sensor, from a sample of the scene: the
    lists are part of the result and as long as the scene makes them."""
    m = 8192
    g = torch.Generator().manual_seed(1)
    means, _, scales, _ = _gaussians(case, m, g, "cpu")
    size = 3.0 * scales.square().mean(-1).sqrt()   # three standard deviations
    if case["kind"] == "lidar":
        r = means.norm(dim=-1)
        reach = torch.rad2deg(size / r).clamp(max=180.0)
        across = (2 * reach / (360.0 / case["columns"] * TILE_WIDTH) + 1).ceil()
        elev = torch.rad2deg(torch.asin(means[:, 2] / r))
        span = (torch.minimum(elev + reach, torch.tensor(16.0)) - torch.maximum(elev - reach, torch.tensor(-26.0)))
        down = (span.clamp(min=0) / (42.0 / math.ceil(case["beams"] / TILE_HEIGHT)) + 1).ceil()
        tiles = across * down * (span > 0)
    else:
        turned = means if case["sensors"] == 1 else torch.stack([-means[:, 1], -means[:, 2], means[:, 0]], -1)
        x, y, z = turned.unbind(-1)
        f, W, H = 0.625 * case["width"], case["width"], case["height"]
        seen = z > 0.01
        z = z.clamp(min=0.01)
        reach = f * size / z + 1.0
        u, v = f * x / z + W / 2, f * y / z + H / 2
        w = (torch.minimum(u + reach, torch.tensor(float(W))) - (u - reach).clamp(min=0)).clamp(min=0)
        h = (torch.minimum(v + reach, torch.tensor(float(H))) - (v - reach).clamp(min=0)).clamp(min=0)
        tiles = (w / TILE_SIZE + 1) * (h / TILE_SIZE + 1) * ((w > 0) & (h > 0) & seen)
    return float((tiles > 0).float().mean()), float(tiles.mean()) * case["n"]


def work(case):
    C, n = case["sensors"], case["n"]
    if case["kind"] == "points":
        pixels = C * case["beams"] * case["columns"]
        # points in (azimuth, elevation and the five values), ids and flatten ids out, the image out
        return {"bytes": C * n * (20 + 12) + pixels * 20, "flops": C * n * 8}
    seen, entries = _estimate(case)
    lidar, ch = case["kind"] == "lidar", _channels(case)
    pixels = C * (case["beams"] * case["columns"] if lidar else case["width"] * case["height"])
    params = n * (3 + 4 + 3 + 1) + math.prod(_colour_shape(case, n))
    rows = C * n * (1.0 if lidar or not case["packed"] else seen)
    per_row = (2 + 2 + 1 + 3 + 3 + 2 + 1) if lidar else (2 + 2 + 1 + 3 + 2 + 1 + 1) + (4 if case["packed"] else 0)
    floats = params + (3 * n if case["moving"] else 0) + rows * per_row + C * entries * 3
    floats += pixels * (ch + 1 + (4 + 3 if lidar else 1))
    # a sample blends the entries that reach it until it is opaque: up to about sixty of them
    tiles = pixels / (TILE_WIDTH * TILE_HEIGHT)
    blended = pixels * min(60.0, 0.5 * C * entries / tiles)
    flops = blended * ((48 if lidar else 22) + 2 * ch) + C * n * 400
    if case["train"]:
        floats += 2 * params + pixels * (ch + 3) + rows * 3
        flops += blended * (90 + 4 * ch) + C * n * 800
    return {"bytes": 4 * floats, "flops": flops}


def tolerance(case):
    if case["kind"] == "points":
        return "exact"
    # 32-bit sums over up to a few hundred blended entries; `max` leaves room for a sample at which two
    # correct evaluations stop, skip or take an entry differently because a threshold falls between them
    if not case["train"]:
        return {"rel": 1e-4, "max": 0.05}
    # Gradients are sums of terms of either sign, largest by far for the few Gaussians next to a sensor:
    # the order of the additions alone (atomics) moves them by 1e-4 from run to run.
    return {"rel": 5e-4, "max": 0.05}
