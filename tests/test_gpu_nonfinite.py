"""Values that are not finite stay where they belong: a sample takes them only from a Gaussian that it blends,
and a Gaussian's gradient only from a sample that blends it - whatever else the same warp is working on."""

import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")


def _camera(channels, packed, cameras=1, mode="RGB"):
    import splatad_b200
    from splatad_b200 import scenes
    s = {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in scenes.config1(N=2_003, packed=packed).items()}
    g = torch.Generator(device=DEV).manual_seed(channels)
    s.update(sh_degree=None, render_mode=mode, width=321, height=203, scales=s["scales"] * (3.0 if cameras == 1 else 9.0),
             colors=torch.rand(2_003, channels, generator=g, device=DEV))
    s["Ks"] = torch.tensor([[[200.0, 0.0, 160.5], [0.0, 200.0, 101.5], [0.0, 0.0, 1.0]]], device=DEV)
    for k in ("viewmats", "Ks", "linear_velocity", "angular_velocity", "rolling_shutter_time"):
        s[k] = s[k].repeat(cameras, *[1] * (s[k].dim() - 1))

    def run(colors, weights=None, **kw):
        p = {k: s[k].clone().requires_grad_(True) for k in ("means", "quats", "scales", "opacities")}
        p["colors"] = colors.clone().requires_grad_(True)
        image, alpha, meta = splatad_b200.rasterization(**{**s, **p, **kw})
        # Gaussians of many tiles: their number, 273 a camera, decides how many pixels a lane draws
        assert cameras == 1 or meta["flatten_ids"].numel() > 15 * int((meta["tiles_per_gauss"] > 0).sum())
        torch.autograd.backward([image, alpha], [torch.ones_like(image) if weights is None else weights, torch.ones_like(alpha)])
        return image.detach(), {k: v.grad for k, v in p.items()}

    return run, s["colors"]


def _lidar(features, columns):
    import splatad_b200
    from splatad_b200 import scenes
    cfg = scenes.config0() if columns == 512 else scenes.config2(N=30_001)
    s = {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in cfg.items()}
    g = torch.Generator(device=DEV).manual_seed(features)
    colors = torch.rand(1, s["means"].shape[0], features, generator=g, device=DEV)

    def run(colors, weights=None, **kw):
        p = {k: s[k].clone().requires_grad_(True) for k in ("means", "quats", "scales", "opacities")}
        p["lidar_features"] = colors.clone().requires_grad_(True)
        image, alpha, alpha_sum, _ = splatad_b200.lidar_rasterization(**{**s, **p, **kw})
        torch.autograd.backward([image, alpha, alpha_sum],
                                [torch.ones_like(image) if weights is None else weights, torch.ones_like(alpha),
                                 torch.ones_like(alpha_sum)])
        p["colors"] = p.pop("lidar_features")
        return image.detach(), {k: v.grad for k, v in p.items()}

    return run, colors


_CASES = [("camera", 3, False), ("camera", 3, True), ("camera", 13, False), ("camera", 30, True),
          ("camera", 7, True, 6), ("camera", 13, False, 6), ("camera", 20, False, 6), ("camera", 3, False, 12), ("camera", 3, True, 24),
          ("lidar", 4, 512), ("lidar", 16, 512), ("lidar", 4, 1800), ("lidar", 16, 1800), ("lidar", 30, 1800)]


def _setup(kind, *args):
    return _camera(*args) if kind == "camera" else _lidar(*args)


def _per_row(t):
    return t.reshape(t.shape[-2], -1) if t.dim() == 3 else t.reshape(t.shape[0], -1)


def _close(got, want, tol):
    assert float((got - want).norm()) <= tol * max(float(want.norm()), 1e-30)


@pytest.mark.parametrize("case", _CASES, ids=str)
@pytest.mark.parametrize("value", [INF, NAN])
def test_a_colour_that_is_not_finite_reaches_its_own_samples_only(case, value):
    run, colors = _setup(*case)
    a = case[1]
    rows = colors.view(-1, a)
    clean, grads = run(colors)
    seen = (grads["colors"].reshape(-1, a).abs().sum(-1) > 0).nonzero()[:, 0]
    bad = int(seen[len(seen) // 2])
    # the samples that blend it: those that a colour of its own reaches
    marker = torch.zeros_like(rows)
    marker[bad] = 1.0
    weight, _ = run(marker.view_as(colors))
    reached = weight[..., 0] > 0
    assert 0 < int(reached.sum()) < reached.numel()
    spoilt = rows.clone()
    spoilt[bad] = value
    image, _ = run(spoilt.view_as(colors))
    finite = torch.isfinite(image[..., :a]).all(-1)
    assert torch.equal(finite, ~reached)
    # 32-bit rounding of the same sums, in whichever way the rest of the tile is worked out
    _close(image[~reached], clean[~reached], 1e-6)


@pytest.mark.parametrize("case", _CASES, ids=str)
@pytest.mark.parametrize("value", [INF, NAN])
def test_a_cotangent_that_is_not_finite_reaches_its_own_gaussians_only(case, value):
    run, colors = _setup(*case)
    image, _ = run(colors)
    at = (0, image.shape[1] // 2, image.shape[2] // 2)
    alone = torch.zeros_like(image)
    alone[at] = 1.0
    _, only = run(colors, alone)
    mine = _per_row(only["colors"]).abs().sum(-1) > 0      # the Gaussians that this sample blends
    assert 0 < int(mine.sum()) < mine.numel()
    without, spoilt = torch.ones_like(image), torch.ones_like(image)
    without[at] = 0.0
    spoilt[at] = value
    _, want = run(colors, without)
    _, got = run(colors, spoilt)
    assert torch.equal(torch.isfinite(_per_row(got["colors"])).all(-1), ~mine)
    for name in ("means", "quats", "scales", "opacities"):
        g, w = _per_row(got[name])[~mine], _per_row(want[name])[~mine]
        assert torch.isfinite(g).all(), name
        _close(g, w, 5e-4)        # sums in another order (atomics): 1e-4 from run to run


@pytest.mark.parametrize("channels", [3, 13])
@pytest.mark.parametrize("what", ["opacities", "means2d", "conics", "pix_vels", "one row", "flat conic"])
def test_a_nan_in_the_geometry_is_blended_with_the_capped_alpha(what, channels):
    """As in the reference, whose minimum of the cap and a NaN is the cap, and as in the oracle."""
    import numpy as np
    from gpu_util import assert_close, n, t
    from oracle import composite
    from splatad_b200 import ops
    from test_gpu_composite import _camera_case
    H = 1 if what == "one row" else 60
    c = _camera_case(1, 300, 100, H, 16, channels, 5)
    if what == "flat conic":                       # and opaque enough around it that pixels have stopped before
        c["conics"][:, ::3] = 0.0
        c["opacities"][:] = 0.6
    elif what != "one row":
        c[what][:, ::29] = float("nan")
    args = [n(c[k]) for k in ("means2d", "conics", "colors", "opacities", "pix_vels", "rs")]
    tail = (None, c["W"], c["H"], c["ts"], c["offsets"], c["flatten_ids"])
    ref = composite.rasterize_to_pixels_fwd(*args, *tail)
    leaves = {k: t(c[k]).requires_grad_(True) for k in ("means2d", "conics", "colors", "opacities", "pix_vels")}
    image, alphas = ops.rasterize_to_pixels(
        leaves["means2d"], leaves["conics"], leaves["colors"], leaves["opacities"], leaves["pix_vels"], c["W"], c["H"], c["ts"],
        t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), t(c["rs"]))
    sure = ~ref["ambiguous"]
    assert sure.mean() > 0.95 and ref["contributing"] > c["W"] * c["H"] // 2
    assert_close("colors", n(image), ref["render_colors"], 1e-4, 1e-5, mask=sure[..., None])
    assert_close("alphas", n(alphas), ref["render_alphas"], 1e-4, 1e-5, mask=sure[..., None])
    mask = sure.astype(np.float32)
    (image * t(mask)[..., None]).sum().backward()
    f64 = composite.rasterize_to_pixels_fwd(*args, *tail, dtype=np.float64)
    want = composite.rasterize_to_pixels_bwd(*args, *tail, f64["render_alphas"], f64["last_ids"],
                                             np.broadcast_to(mask[..., None], n(image).shape).astype(np.float64),
                                             np.zeros(n(alphas).shape))
    for k in ("means2d", "conics", "colors", "opacities", "pix_vels"):
        got, ref_k = n(leaves[k].grad), want["v_" + k]
        assert np.array_equal(np.isfinite(got), np.isfinite(ref_k)), k
        got, ref_k = np.nan_to_num(got).astype(np.float64), np.nan_to_num(ref_k)
        assert np.linalg.norm(got - ref_k) <= 2e-3 * max(np.linalg.norm(ref_k), 1e-20), k


@pytest.mark.parametrize("C,channels,mode,spread", [(1600, 3, "x", 0), (1600, 3, "x", 8), (1600, 7, "x", 0), (1600, 13, "x", 0), (1600, 18, "x", 0),
                                                    (3200, 4, "y", 0), (6400, 3, "y", 0), (6400, 3, "x", 5), (1000, 30, "x", 0)])
@pytest.mark.parametrize("value", [INF, NAN])
def test_a_colour_that_is_not_finite_and_hidden_reaches_nothing(C, channels, mode, spread, value):
    """One half of every tile stops early; a Gaussian behind that has a colour that is not finite and does not reach the other half,
    which blends one further behind. Nobody blends it: image and gradients are those of a finite colour and its own
    gradients are zero, also where the backward pass works on both halves at once and the forward pass on each by itself."""
    from gpu_util import t
    from splatad_b200 import ops
    layers, bad, last = 150, 150, 151
    along, across = (0, 1) if mode == "x" else (1, 0)
    means = torch.full((layers + 2, 2), 8.0)
    means[:bad, along], means[bad, along], means[last, along] = 4.0, 3.0, 13.0
    tight, wide = torch.full((layers + 2,), 0.3), torch.full((layers + 2,), 1e-4)   # (1/px^2) along the split and across it
    tight[bad], tight[last] = 4.0, 1.0
    conics = torch.zeros(layers + 2, 3)
    conics[:, 0], conics[:, 2] = (tight, wide) if mode == "x" else (wide, tight)
    g = torch.Generator().manual_seed(channels)
    colors = torch.rand(layers + 2, channels, generator=g)
    opacities = torch.full((layers + 2,), 0.95)
    n = layers + 2
    fixed = dict(means2d=means, conics=conics, opacities=opacities, pix_vels=torch.zeros(n, 2))
    offsets = t(torch.arange(C)[:, None, None] * n, torch.int32)
    ids = t(torch.arange(C * n), torch.int32)
    ids._splatad_spread, ids._splatad_count = float(spread), 10**7   # as if the Gaussians covered as many tiles
    weights = [t(torch.randn(1, 16, 16, k, generator=g)).expand(C, -1, -1, -1).contiguous() for k in (channels, 1)]

    def run(bad_colour):
        c = colors.clone()
        c[bad] = bad_colour
        p = {k: t(v)[None].expand(C, *v.shape).contiguous().requires_grad_(True) for k, v in dict(colors=c, **fixed).items()}
        out = ops.rasterize_to_pixels(p["means2d"], p["conics"], p["colors"], p["opacities"], p["pix_vels"], 16, 16, 16,
                                      offsets, ids, torch.zeros(C, device=DEV), absgrad=True)
        torch.autograd.backward(out, weights)
        return [o.detach() for o in out], {**{k: v.grad for k, v in p.items()}, "absolute": p["means2d"].absgrad}

    out, want = run(0.5)
    assert float(want["colors"][:, bad].abs().max()) == 0.0 and float(want["colors"][:, last].abs().min()) > 0.0
    spoilt, got = run(value)
    for a, b in zip(out, spoilt):
        _close(b, a, 1e-6)                 # as above: in whichever way the tile is worked out
    for k in want:
        assert torch.isfinite(got[k]).all() and float(got[k][:, bad].abs().max()) == 0.0, k
        _close(got[k], want[k], 1e-5)      # sums over a tile in another order


@pytest.mark.parametrize("C,channels", [(1, 5), (9, 5), (1, 18), (9, 18)])
@pytest.mark.parametrize("coordinate", [0, 1, 3])
@pytest.mark.parametrize("value", [NAN, INF])
def test_a_lidar_point_that_is_not_finite_blends_the_first_entry(C, channels, coordinate, value):
    """A point without an azimuth, an elevation or a time, among points that have them and in a patch of nothing else: as in the
    oracle it takes the first entry of its list with the capped alpha and a range that is not a number, in scans whose
    warps share a patch and in those whose do not. The Gaussians that it does not blend get the gradients of the others."""
    import numpy as np
    from gpu_util import assert_close, n, t
    from oracle import composite
    from splatad_b200 import ops
    from test_gpu_composite import _lidar_case
    H, W, tw, th = 64, 320, 32, 8          # 640 patches a sensor
    c = _lidar_case(C, 600, H, W, tw, th, channels, 11 * C + channels)
    c["pts"][:, 5, 7, 2] = 20.0            # alone in its patch
    c["pts"][:, 5, 7, coordinate] = value
    c["pts"][:, 32:36, 200:208, 2] = 20.0  # a whole patch
    c["pts"][:, 32:36, 200:208, coordinate] = value
    spoilt = ~torch.isfinite(c["pts"]).all(-1).numpy()
    keys = ("means2d", "conics", "feats", "opacities", "pix_vels", "dcomp")
    args = [n(c[k]) for k in keys] + [None, n(c["pts"]), W, H, tw, th, c["offsets"], c["flatten_ids"], True, 0.5]
    ref = composite.rasterize_to_points_fwd(*args, amb_tol=1e-4)
    assert np.isnan(ref["render_colors"][spoilt][:, -1]).all() and (ref["render_alphas"][spoilt] > 0.9).all()
    leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
    image, alphas, sums, medians = ops.rasterize_to_points(
        *(leaves[k] for k in keys), t(c["pts"]), W, H, tw, th, t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), True, 0.5)
    sure = ~ref["ambiguous"] | spoilt
    for got, want in ((image, ref["render_colors"]), (alphas, ref["render_alphas"]), (sums, ref["alpha_sum"])):
        got, want = n(got), want.reshape(n(got).shape)
        assert np.array_equal(np.isnan(got[sure]), np.isnan(want[sure]))
        assert_close("points", np.nan_to_num(got), np.nan_to_num(want), 2e-4, 2e-5, mask=sure[..., None])
    torch.autograd.backward([image, alphas], [torch.ones_like(image), torch.ones_like(alphas)])
    f64 = composite.rasterize_to_points_fwd(*args, dtype=np.float64)
    want = composite.rasterize_to_points_bwd(*args, f64["render_alphas"], f64["last_ids"], np.ones(n(image).shape),
                                             np.ones(n(alphas).shape), np.zeros(n(alphas).shape))
    same = (f64["last_ids"] == ref["last_ids"]).mean()
    assert same > 0.99
    for k, name in zip(keys, ("v_means2d", "v_conics", "v_colors", "v_opacities", "v_pix_vels", "v_depth_comps")):
        got, ref_k = n(leaves[k].grad), want[name].reshape(leaves[k].shape)
        assert np.array_equal(np.isfinite(got), np.isfinite(ref_k)), k
