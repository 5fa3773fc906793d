"""Values that are not finite stay where they belong: a sample takes them only from a Gaussian that it blends,
and a Gaussian's gradient only from a sample that blends it - whatever else the same warp is working on."""

import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")


def _camera(channels, packed, mode="RGB"):
    import splatad_b200
    from splatad_b200 import scenes
    s = {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in scenes.config1(N=2_003, packed=packed).items()}
    g = torch.Generator(device=DEV).manual_seed(channels)
    s.update(sh_degree=None, render_mode=mode, width=321, height=203, scales=s["scales"] * 3.0,
             colors=torch.rand(2_003, channels, generator=g, device=DEV))
    s["Ks"] = torch.tensor([[[200.0, 0.0, 160.5], [0.0, 200.0, 101.5], [0.0, 0.0, 1.0]]], device=DEV)

    def run(colors, weights=None, **kw):
        p = {k: s[k].clone().requires_grad_(True) for k in ("means", "quats", "scales", "opacities")}
        p["colors"] = colors.clone().requires_grad_(True)
        image, alpha, _ = splatad_b200.rasterization(**{**s, **p, **kw})
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
          ("lidar", 4, 512), ("lidar", 16, 512), ("lidar", 4, 1800), ("lidar", 16, 1800), ("lidar", 30, 1800)]


def _setup(kind, a, b):
    return _camera(a, b) if kind == "camera" else _lidar(a, b)


def _per_row(t):
    return t.reshape(t.shape[-2], -1) if t.dim() == 3 else t.reshape(t.shape[0], -1)


def _close(got, want, tol):
    assert float((got - want).norm()) <= tol * max(float(want.norm()), 1e-30)


@pytest.mark.parametrize("kind,a,b", _CASES)
@pytest.mark.parametrize("value", [INF, NAN])
def test_a_colour_that_is_not_finite_reaches_its_own_samples_only(kind, a, b, value):
    run, colors = _setup(kind, a, b)
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


@pytest.mark.parametrize("kind,a,b", _CASES)
@pytest.mark.parametrize("value", [INF, NAN])
def test_a_cotangent_that_is_not_finite_reaches_its_own_gaussians_only(kind, a, b, value):
    run, colors = _setup(kind, a, b)
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
