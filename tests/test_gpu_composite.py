"""Parity of the compositing kernels (rasterize_to_pixels / rasterize_to_points, forward and
backward, through the C ABI) against the C oracle.

Forward tolerance: 1e-4 relative + 1e-5 absolute on every pixel whose threshold decisions are
not within 2e-5 (relative) of flipping; the oracle flags those (a different but equally valid
floating-point evaluation order may include or exclude one more Gaussian there) and their
fraction is asserted to be small. Ranges (depth) are also checked to 1 mm.
Backward tolerance: 1e-3 relative against the float64 oracle.
"""

import math

import numpy as np
import pytest
import torch

from gpu_util import DEV, assert_close, launched, n, rel_l2, t

pytestmark = pytest.mark.gpu


def _camera_case(C, N, W, H, ts, channels, seed, rs_time=0.03, sigma_px=(2.0, 14.0)):
    from oracle import isect
    g = torch.Generator().manual_seed(seed)
    means2d = (torch.rand(C, N, 2, generator=g) * 1.1 - 0.05) * torch.tensor([W, H])
    sig = torch.rand(C, N, 2, generator=g) * (sigma_px[1] - sigma_px[0]) + sigma_px[0]
    rho = torch.rand(C, N, generator=g) * 1.2 - 0.6
    cov = torch.stack([sig[..., 0] ** 2, rho * sig[..., 0] * sig[..., 1], rho * sig[..., 0] * sig[..., 1],
                       sig[..., 1] ** 2], -1).reshape(C, N, 2, 2)
    inv = torch.linalg.inv(cov)
    conics = torch.stack([inv[..., 0, 0], inv[..., 0, 1], inv[..., 1, 1]], -1).contiguous()
    opac = torch.rand(C, N, generator=g) * 0.95 + 0.04
    opac[:, ::13] = 1.0  # exercises the 0.999 cap
    colors = torch.randn(C, N, channels, generator=g)
    pix_vels = torch.randn(C, N, 2, generator=g) * 40
    depths = torch.rand(C, N, generator=g) * 50 + 0.5
    rs = torch.full((C,), rs_time)
    radii = (3 * sig + pix_vels.abs() * 0.5 * rs_time).to(torch.int32)
    tw, th = math.ceil(W / ts), math.ceil(H / ts)
    _, ids, flat = isect.isect_tiles(n(means2d), n(radii), n(depths), ts, tw, th)
    offs = isect.isect_offset_encode(ids, C, tw, th)
    return dict(means2d=means2d, conics=conics, colors=colors, opacities=opac, pix_vels=pix_vels, rs=rs,
                offsets=offs, flatten_ids=flat, W=W, H=H, ts=ts)


def _check_fwd(label, got_c, got_a, ref, depth_channel=None):
    amb = ref["ambiguous"]
    frac = amb.mean()
    assert frac < 0.02, f"{label}: {frac:.3%} of the pixels are within tolerance of a threshold"
    ok = ~amb
    assert_close(label + " colors", got_c, ref["render_colors"], 1e-4, 1e-5, mask=ok[..., None])
    assert_close(label + " alphas", got_a, ref["render_alphas"], 1e-4, 1e-5, mask=ok[..., None])
    if depth_channel is not None:
        d = np.abs(got_c[..., depth_channel] - ref["render_colors"][..., depth_channel])[ok]
        lim = 1e-3 + 1e-4 * np.abs(ref["render_colors"][..., depth_channel])[ok]
        assert (d <= lim).all(), f"{label}: range off by {d.max()} m"


@pytest.mark.parametrize("channels", [1, 3, 4, 5, 17, 32])
@pytest.mark.parametrize("with_bg", [False, True])
def test_rasterize_to_pixels_fwd(channels, with_bg):
    from oracle import composite
    from splatad_b200 import ops
    c = _camera_case(2, 3000, 200, 136, 16, channels, 100 + channels)
    bg = torch.rand(2, channels) if with_bg else None
    ref = composite.rasterize_to_pixels_fwd(n(c["means2d"]), n(c["conics"]), n(c["colors"]), n(c["opacities"]),
                                            n(c["pix_vels"]), n(c["rs"]), n(bg), c["W"], c["H"], c["ts"],
                                            c["offsets"], c["flatten_ids"])
    out_c, out_a = ops.rasterize_to_pixels(t(c["means2d"]), t(c["conics"]), t(c["colors"]), t(c["opacities"]),
                                           t(c["pix_vels"]), c["W"], c["H"], c["ts"],
                                           t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32),
                                           t(c["rs"]), backgrounds=t(bg))
    assert ref["contributing"] > 10 * c["W"] * c["H"]
    _check_fwd(f"pixels ch={channels} bg={with_bg}", n(out_c), n(out_a), ref)


def test_rasterize_to_pixels_many_channels_and_odd_tile():
    """> 32 channels are rendered in chunks; tile sizes whose square is not a warp multiple work."""
    from oracle import composite
    from splatad_b200 import ops
    c = _camera_case(1, 800, 70, 50, 6, 40, 7)
    ref = composite.rasterize_to_pixels_fwd(n(c["means2d"]), n(c["conics"]), n(c["colors"]), n(c["opacities"]),
                                            n(c["pix_vels"]), n(c["rs"]), None, c["W"], c["H"], c["ts"],
                                            c["offsets"], c["flatten_ids"])
    out_c, out_a = ops.rasterize_to_pixels(t(c["means2d"]), t(c["conics"]), t(c["colors"]), t(c["opacities"]),
                                           t(c["pix_vels"]), c["W"], c["H"], c["ts"],
                                           t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), t(c["rs"]))
    _check_fwd("pixels 40 channels tile 6", n(out_c), n(out_a), ref)


@pytest.mark.parametrize("channels", [3, 20])
def test_rasterize_to_pixels_largest_tile(channels):
    """32 x 32 tiles are blocks of 1024 threads: the forward kernels run at any channel count, the
    backward kernels while their registers allow it and say so otherwise."""
    from oracle import composite
    from splatad_b200 import ops
    c = _camera_case(1, 1500, 100, 70, 32, channels, 70 + channels)
    ref = composite.rasterize_to_pixels_fwd(n(c["means2d"]), n(c["conics"]), n(c["colors"]), n(c["opacities"]),
                                            n(c["pix_vels"]), n(c["rs"]), None, c["W"], c["H"], c["ts"],
                                            c["offsets"], c["flatten_ids"])
    leaves = {k: t(c[k]).requires_grad_(True) for k in ("means2d", "conics", "colors", "opacities", "pix_vels")}
    out_c, out_a = ops.rasterize_to_pixels(leaves["means2d"], leaves["conics"], leaves["colors"], leaves["opacities"],
                                           leaves["pix_vels"], c["W"], c["H"], c["ts"],
                                           t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), t(c["rs"]))
    _check_fwd(f"pixels tile 32 ch={channels}", n(out_c), n(out_a), ref)
    loss = out_c.sum() + out_a.sum()
    if channels == 3:
        loss.backward()
        assert float(leaves["colors"].grad.abs().sum()) > 0
    else:
        with pytest.raises(ValueError, match="1024 threads"):
            loss.backward()


def _grad_check(label, got, want, rel=1e-3):
    got, want = n(got).astype(np.float64), np.asarray(want, dtype=np.float64)
    rms = float(np.sqrt(np.mean(want ** 2)))
    e = rel_l2(got, want)
    assert e < rel, f"{label}: relative L2 error {e:.3e}"
    assert_close(label, got, want, rel, 2 * rel * rms, max_bad_frac=2e-3)


@pytest.mark.parametrize("channels,with_bg,absgrad", [(3, False, True), (4, True, False), (17, False, False)])
def test_rasterize_to_pixels_bwd(channels, with_bg, absgrad):
    from oracle import composite
    from splatad_b200 import ops
    c = _camera_case(2, 2000, 160, 120, 16, channels, 200 + channels)
    bg = torch.rand(2, channels) if with_bg else None
    g = torch.Generator().manual_seed(3)
    v_c = torch.randn(2, c["H"], c["W"], channels, generator=g)
    v_a = torch.randn(2, c["H"], c["W"], 1, generator=g)
    leaves = {k: t(c[k]).requires_grad_(True) for k in ("means2d", "conics", "colors", "opacities", "pix_vels")}
    bg_g = t(bg).requires_grad_(True) if with_bg else None
    ref_f = composite.rasterize_to_pixels_fwd(n(c["means2d"]), n(c["conics"]), n(c["colors"]), n(c["opacities"]),
                                              n(c["pix_vels"]), n(c["rs"]), n(bg), c["W"], c["H"], c["ts"],
                                              c["offsets"], c["flatten_ids"], dtype=np.float64)
    # only pixels whose include/exclude decisions are unambiguous take part in the comparison
    f32 = composite.rasterize_to_pixels_fwd(n(c["means2d"]), n(c["conics"]), n(c["colors"]), n(c["opacities"]),
                                            n(c["pix_vels"]), n(c["rs"]), n(bg), c["W"], c["H"], c["ts"],
                                            c["offsets"], c["flatten_ids"], amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    assert same.mean() > 0.97
    mask = t(same[..., None].astype(np.float32))
    out_c, out_a = ops.rasterize_to_pixels(leaves["means2d"], leaves["conics"], leaves["colors"],
                                           leaves["opacities"], leaves["pix_vels"], c["W"], c["H"], c["ts"],
                                           t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32),
                                           t(c["rs"]), backgrounds=bg_g, absgrad=absgrad)
    ((out_c * t(v_c) * mask).sum() + (out_a * t(v_a) * mask).sum()).backward()
    mk = same[..., None].astype(np.float64)
    ref = composite.rasterize_to_pixels_bwd(n(c["means2d"]), n(c["conics"]), n(c["colors"]), n(c["opacities"]),
                                            n(c["pix_vels"]), n(c["rs"]), n(bg), c["W"], c["H"], c["ts"],
                                            c["offsets"], c["flatten_ids"], ref_f["render_alphas"],
                                            ref_f["last_ids"], n(v_c) * mk, n(v_a) * mk, absgrad=absgrad)
    _grad_check("pixels v_means2d", leaves["means2d"].grad, ref["v_means2d"])
    _grad_check("pixels v_conics", leaves["conics"].grad, ref["v_conics"])
    _grad_check("pixels v_colors", leaves["colors"].grad, ref["v_colors"])
    _grad_check("pixels v_opacities", leaves["opacities"].grad, ref["v_opacities"])
    _grad_check("pixels v_pix_vels", leaves["pix_vels"].grad, ref["v_pix_vels"])
    if absgrad:
        _grad_check("pixels absgrad", leaves["means2d"].absgrad, ref["v_means2d_abs"])
    if with_bg:
        want_bg = (n(v_c) * mk * (1.0 - ref_f["render_alphas"])).sum(axis=(1, 2))
        _grad_check("pixels v_backgrounds", bg_g.grad, want_bg)


def _lidar_case(C, N, H, W, tw, th, channels, seed, sweep=0.1):
    from oracle import isect
    from splatad_b200 import scenes
    g = torch.Generator().manual_seed(seed)
    elev = torch.linspace(-20.0, 12.0, H)
    az_res = 360.0 / W
    pts = torch.cat([scenes.lidar_sensor(elev, W, g, sweep_time=sweep) for _ in range(C)], 0)
    pts[..., :2] += torch.randn(C, H, W, 2, generator=g) * 0.01
    pts[..., 2] = pts[..., 2] * (torch.rand(C, H, W, generator=g) > 0.1)  # ~10 % of the points have no return
    means2d = torch.stack([torch.rand(C, N, generator=g) * 360 - 180, torch.rand(C, N, generator=g) * 36 - 22], -1)
    sig = torch.rand(C, N, 2, generator=g) * torch.tensor([4.0, 2.0]) + torch.tensor([0.5, 0.3])
    rho = torch.rand(C, N, generator=g) * 1.2 - 0.6
    cov = torch.stack([sig[..., 0] ** 2, rho * sig[..., 0] * sig[..., 1], rho * sig[..., 0] * sig[..., 1],
                       sig[..., 1] ** 2], -1).reshape(C, N, 2, 2)
    inv = torch.linalg.inv(cov)
    conics = torch.stack([inv[..., 0, 0], inv[..., 0, 1], inv[..., 1, 1]], -1).contiguous()
    opac = torch.rand(C, N, generator=g) * 0.95 + 0.04
    opac[:, ::13] = 1.0
    depths = torch.rand(C, N, generator=g) * 80 + 1
    feats = torch.randn(C, N, channels, generator=g)
    feats[..., -1] = depths
    pix_vels = torch.randn(C, N, 3, generator=g) * torch.tensor([20.0, 5.0, 3.0])
    dcomp = torch.randn(C, N, 2, generator=g) * 0.05
    radii = 3 * sig + pix_vels[..., :2].abs() * 0.5 * sweep
    eb = scenes.elevation_boundaries(elev, th)
    res = az_res * tw
    _, ids, flat = isect.isect_lidar_tiles(n(means2d), n(radii), n(depths), n(eb), res, -180.0)
    n_az = math.ceil(360 / res)
    offs = isect.isect_offset_encode(ids, C, n_az, len(eb) - 1)
    return dict(means2d=means2d, conics=conics, feats=feats, opacities=opac, pix_vels=pix_vels, dcomp=dcomp,
                pts=pts, offsets=offs, flatten_ids=flat, W=W, H=H, tw=tw, th=th)


@pytest.mark.parametrize("channels", [2, 5, 17, 32])
@pytest.mark.parametrize("asum", [False, True])
def test_rasterize_to_points_fwd(channels, asum):
    from oracle import composite
    from splatad_b200 import ops
    c = _lidar_case(2, 4000, 32, 512, 32, 8, channels, 300 + channels)
    ref = composite.rasterize_to_points_fwd(n(c["means2d"]), n(c["conics"]), n(c["feats"]), n(c["opacities"]),
                                            n(c["pix_vels"]), n(c["dcomp"]), None, n(c["pts"]), c["W"], c["H"],
                                            c["tw"], c["th"], c["offsets"], c["flatten_ids"], asum, 0.5)
    out_c, out_a, out_s, out_m = ops.rasterize_to_points(
        t(c["means2d"]), t(c["conics"]), t(c["feats"]), t(c["opacities"]), t(c["pix_vels"]), t(c["dcomp"]),
        t(c["pts"]), c["W"], c["H"], c["tw"], c["th"], t(c["offsets"], torch.int32),
        t(c["flatten_ids"], torch.int32), asum, 0.5)
    assert ref["contributing"] > 5 * c["W"] * c["H"]
    label = f"points ch={channels} asum={asum}"
    _check_fwd(label, n(out_c), n(out_a), ref, depth_channel=channels - 1)
    ok = ~ref["ambiguous"][..., None]
    assert_close(label + " median", n(out_m), ref["median_depths"], 1e-4, 1e-3, mask=ok)
    if asum:
        assert_close(label + " alpha_sum", n(out_s), ref["alpha_sum"], 1e-4, 1e-5, mask=ok)
    else:
        assert out_s is None
    # points without a return render nothing
    dead = n(c["pts"])[..., 2] <= 0
    assert dead.any() and np.all(n(out_c)[dead] == 0) and np.all(n(out_a)[dead] == 0)


@pytest.mark.parametrize("channels,asum,absgrad", [(5, True, True), (17, False, False), (4, True, False)])
def test_rasterize_to_points_bwd(channels, asum, absgrad):
    from oracle import composite
    from splatad_b200 import ops
    c = _lidar_case(2, 3000, 32, 256, 32, 8, channels, 400 + channels)
    g = torch.Generator().manual_seed(4)
    C, H, W = 2, c["H"], c["W"]
    v_c = torch.randn(C, H, W, channels, generator=g)
    v_a = torch.randn(C, H, W, 1, generator=g)
    v_s = torch.randn(C, H, W, 1, generator=g)
    keys = ("means2d", "conics", "feats", "opacities", "pix_vels", "dcomp")
    args64 = [n(c[k]) for k in keys]
    ref_f = composite.rasterize_to_points_fwd(*args64, None, n(c["pts"]), W, H, c["tw"], c["th"], c["offsets"],
                                              c["flatten_ids"], asum, 0.5, dtype=np.float64)
    f32 = composite.rasterize_to_points_fwd(*args64, None, n(c["pts"]), W, H, c["tw"], c["th"], c["offsets"],
                                            c["flatten_ids"], asum, 0.5, amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    assert same.mean() > 0.97
    mk = same[..., None].astype(np.float64)
    mask = t(mk)
    leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
    out_c, out_a, out_s, _ = ops.rasterize_to_points(
        leaves["means2d"], leaves["conics"], leaves["feats"], leaves["opacities"], leaves["pix_vels"],
        leaves["dcomp"], t(c["pts"]), W, H, c["tw"], c["th"], t(c["offsets"], torch.int32),
        t(c["flatten_ids"], torch.int32), asum, 0.5, absgrad=absgrad)
    loss = (out_c * t(v_c) * mask).sum() + (out_a * t(v_a) * mask).sum()
    if asum:
        loss = loss + (out_s * t(v_s) * mask).sum()
    loss.backward()
    ref = composite.rasterize_to_points_bwd(*args64, None, n(c["pts"]), W, H, c["tw"], c["th"], c["offsets"],
                                            c["flatten_ids"], asum, 0.5, ref_f["render_alphas"], ref_f["last_ids"],
                                            n(v_c) * mk, n(v_a) * mk, (n(v_s) * mk) if asum else None,
                                            absgrad=absgrad)
    _grad_check("points v_means2d", leaves["means2d"].grad, ref["v_means2d"])
    _grad_check("points v_conics", leaves["conics"].grad, ref["v_conics"])
    _grad_check("points v_features", leaves["feats"].grad, ref["v_colors"])
    _grad_check("points v_opacities", leaves["opacities"].grad, ref["v_opacities"])
    _grad_check("points v_pix_vels", leaves["pix_vels"].grad, ref["v_pix_vels"])
    _grad_check("points v_depth_comps", leaves["dcomp"].grad, ref["v_depth_comps"])
    if absgrad:
        _grad_check("points absgrad", leaves["means2d"].absgrad, ref["v_means2d_abs"])


def test_accumulate_until_points_known_answer():
    """Ten Gaussians stacked on one lidar point at ranges 20..120 m, the point at 85 m, threshold
    0.5 m (the hand-built case of the reference's tests/test_basic.py:1257-1281): the alpha sum
    counts exactly the Gaussians nearer than 84.5 m, and every output has a closed form."""
    from splatad_b200 import ops
    from oracle import isect
    H, W, tw, th = 32, 1800, 64, 4
    elev = torch.linspace(-30.0, 30.0, H)
    az = torch.linspace(-180 + 0.1, 180 - 0.1, W)
    pts = torch.zeros(1, H, W, 4)
    pts[0, :, :, 0] = az[None, :]
    pts[0, :, :, 1] = elev[:, None]
    pi, pj = 16, 900
    pts[0, pi, pj, 2] = 85.0
    N = 10
    means2d = (pts[0, pi, pj, :2] + 0.1).repeat(N, 1)[None]
    conics = torch.tensor([1.0, 0.0, 1.0]).repeat(N, 1)[None]
    depths = torch.linspace(20.0, 120.0, N)[None]
    g = torch.Generator().manual_seed(9)
    opac = torch.rand(1, N, generator=g)
    feats = torch.cat([torch.randn(1, N, 5, generator=g), depths[..., None]], -1)
    radii = torch.ones(1, N, 2)
    eb = torch.linspace(-30.0 - 1e-2, 30.0 + 1e-2, H // th + 1)
    res = 0.2 * tw
    _, ids, flat = isect.isect_lidar_tiles(n(means2d), n(radii), n(depths), n(eb), res, -180.0)
    offs = isect.isect_offset_encode(ids, 1, math.ceil(360 / res), H // th)
    out_c, out_a, out_s, out_m = ops.rasterize_to_points(
        t(means2d), t(conics), t(feats), t(opac), torch.zeros(1, N, 3, device=DEV),
        torch.zeros(1, N, 2, device=DEV), t(pts), W, H, tw, th, t(offs, torch.int32), t(flat, torch.int32),
        True, 0.5)
    # closed form
    alpha = np.minimum(0.999, n(opac)[0].astype(np.float64) * math.exp(-0.5 * (0.1 ** 2 + 0.1 ** 2)))
    T, want_c, want_s, median = 1.0, np.zeros(6), 0.0, 0.0
    for k in range(N):
        if alpha[k] < 1 / 255:
            continue
        nT = T * (1 - alpha[k])
        if nT <= 1e-4:
            break
        want_c += n(feats)[0, k] * alpha[k] * T
        if T > 0.5 >= nT:
            median = float(depths[0, k])
        if float(depths[0, k]) < 85.0 - 0.5:
            want_s += alpha[k]
        T = nT
    assert_close("known answer features", n(out_c)[0, pi, pj], want_c, 1e-4, 1e-5)
    assert_close("known answer alpha", n(out_a)[0, pi, pj, 0], 1 - T, 1e-4, 1e-5)
    assert_close("known answer alpha sum", n(out_s)[0, pi, pj, 0], want_s, 1e-4, 1e-5)
    assert_close("known answer median", n(out_m)[0, pi, pj, 0], median, 1e-5, 1e-5)
    # every other point has range 0: nothing rendered
    others = np.ones((H, W), bool)
    others[pi, pj] = False
    assert np.all(n(out_a)[0, others] == 0) and np.all(n(out_c)[0, others] == 0)


@pytest.mark.parametrize("channels", [1, 5, 32])
def test_rasterize_to_points_split_ranges(channels):
    """Ranges passed as their own array give the same render and the same gradients as ranges
    concatenated to the features as last channel (the reference's layout, gsplat/rendering.py:779)."""
    from splatad_b200 import ops
    c = _lidar_case(2, 3000, 32, 256, 32, 8, channels, 500 + channels)
    g = torch.Generator().manual_seed(5)
    C, H, W = 2, c["H"], c["W"]
    v = [t(torch.randn(C, H, W, k, generator=g)) for k in (channels, 1, 1)]
    common = lambda L: (L["opacities"], L["pix_vels"], L["dcomp"], t(c["pts"]), W, H, c["tw"], c["th"],
                        t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), True, 0.5)
    keys = ("means2d", "conics", "feats", "opacities", "pix_vels", "dcomp")
    A = {k: t(c[k]).requires_grad_(True) for k in keys}
    outs_a = ops.rasterize_to_points(A["means2d"], A["conics"], A["feats"], *common(A))
    B = {k: t(c[k]).requires_grad_(True) for k in keys if k != "feats"}
    B["f"] = t(c["feats"][..., :-1].contiguous()).requires_grad_(True)
    B["r"] = t(c["feats"][..., -1].contiguous()).requires_grad_(True)
    outs_b = ops.rasterize_to_points_split(B["means2d"], B["conics"], B["f"], B["r"], *common(B))
    # same decisions, same arithmetic; the compiler may contract the range accumulation differently
    assert_close("split render", n(outs_b[0]), n(outs_a[0]), 1e-6, 1e-7)
    for a, b in zip(outs_a[1:], outs_b[1:]):
        assert torch.equal(a, b)
    for outs in (outs_a, outs_b):
        (outs[0] * v[0]).sum().add((outs[1] * v[1]).sum()).add((outs[2] * v[2]).sum()).backward()
    for k in ("means2d", "conics", "opacities", "pix_vels", "dcomp"):
        _grad_check(f"split {k}", B[k].grad, n(A[k].grad), rel=1e-5)
    if channels > 1:
        _grad_check("split features", B["f"].grad, n(A["feats"].grad[..., :-1]), rel=1e-5)
    _grad_check("split ranges", B["r"].grad, n(A["feats"].grad[..., -1]), rel=1e-5)


@pytest.mark.parametrize("ts,W,H,channels,absgrad", [(1, 9, 5, 3, False), (5, 33, 21, 4, True), (16, 17, 16, 1, False),
                                                     (16, 15, 2, 8, True), (17, 50, 40, 9, False), (31, 62, 45, 3, True),
                                                     (16, 40, 33, 20, True), (8, 30, 30, 32, False)])
def test_pixels_several_per_thread(ts, W, H, channels, absgrad):
    """Threads draw two or four pixels of a row, warps cover patches of a tile and skip what cannot reach
    them: tile sizes that are no multiple of either, images that end inside a patch or a thread's
    pixels, every channel group, forward and backward against the oracle."""
    from oracle import composite
    from splatad_b200 import ops
    c = _camera_case(1, 900, W, H, ts, channels, 1000 * ts + channels)
    g = torch.Generator().manual_seed(3)
    v_c, v_a = torch.randn(1, H, W, channels, generator=g), torch.randn(1, H, W, 1, generator=g)
    keys = ("means2d", "conics", "colors", "opacities", "pix_vels")
    args = [n(c[k]) for k in keys] + [n(c["rs"]), None, W, H, ts, c["offsets"], c["flatten_ids"]]
    ref_f = composite.rasterize_to_pixels_fwd(*args, dtype=np.float64)
    f32 = composite.rasterize_to_pixels_fwd(*args, amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    assert same.mean() > 0.9
    mask, mk = t(same[..., None].astype(np.float32)), same[..., None].astype(np.float64)
    leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
    out_c, out_a = ops.rasterize_to_pixels(*(leaves[k] for k in keys), W, H, ts, t(c["offsets"], torch.int32),
                                           t(c["flatten_ids"], torch.int32), t(c["rs"]), absgrad=absgrad)
    _check_fwd(f"pixels tile {ts} {W}x{H} ch={channels}", n(out_c), n(out_a), f32)
    torch.autograd.backward([out_c, out_a], [t(v_c) * mask, t(v_a) * mask])
    ref = composite.rasterize_to_pixels_bwd(*args, ref_f["render_alphas"], ref_f["last_ids"], n(v_c) * mk, n(v_a) * mk,
                                            absgrad=absgrad)
    for k in keys:
        _grad_check(f"tile {ts} ch={channels} v_{k}", leaves[k].grad, ref["v_" + k])
    if absgrad:
        _grad_check(f"tile {ts} ch={channels} absgrad", leaves["means2d"].absgrad, ref["v_means2d_abs"])


@pytest.mark.parametrize("C,ts,channels,absgrad", [(24, 16, 3, True), (43, 16, 4, False), (84, 16, 3, False), (86, 16, 4, True),
                                                   (24, 16, 8, True), (43, 16, 7, False), (24, 16, 13, True), (24, 16, 20, False),
                                                   (96, 24, 4, False), (96, 32, 2, True)])
def test_pixels_of_many_tiles(C, ts, channels, absgrad):
    """Frames of many tiles take four and eight pixels of a row per lane: images that end inside a tile, a row of 16-byte
    pieces or a lane's pixels, opacities above the cap, and conics on either side of those whose alphas need care
    (needles, and one that is not positive definite), forward and backward against the oracle."""
    from oracle import composite
    from splatad_b200 import ops
    W, H = (127, 133) if C % 2 else (132, 131)
    c = _camera_case(C, 120, W, H, ts, channels, 1000 * ts + channels)
    for k, rho in enumerate((0.999, 0.99999, 0.9999999, 1.5)):   # 1 - rho^2 against 1e-5
        a, b = c["conics"][:, 2 + k, 0], c["conics"][:, 2 + k, 2]
        c["conics"][:, 2 + k, 1] = rho * torch.sqrt(a * b)
    g = torch.Generator().manual_seed(3)
    v_c, v_a = torch.randn(C, H, W, channels, generator=g), torch.randn(C, H, W, 1, generator=g)
    keys = ("means2d", "conics", "colors", "opacities", "pix_vels")
    args = [n(c[k]) for k in keys] + [n(c["rs"]), None, W, H, ts, c["offsets"], c["flatten_ids"]]
    ref_f = composite.rasterize_to_pixels_fwd(*args, dtype=np.float64)
    f32 = composite.rasterize_to_pixels_fwd(*args, amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    assert same.mean() > 0.9
    # of a form that nearly vanishes or is negative somewhere, the sign and the size hang on the last bits: the pixels
    # within reach of its rounding are left out (relative to its terms, as the kernel and the oracle sum them)
    j, i = np.meshgrid(np.arange(W) + 0.5, np.arange(H) + 0.5)
    roll = n(c["rs"])[:, None, None] * ((i - 0.5) / (H - 1) - 0.5)
    for k in range(2, 6):
        m, v, q = (n(c[key])[:, k].astype(np.float64) for key in ("means2d", "pix_vels", "conics"))
        dx = m[:, 0, None, None] + roll * v[:, 0, None, None] - j
        dy = m[:, 1, None, None] + roll * v[:, 1, None, None] - i
        size = 0.5 * (q[:, 0, None, None] * dx * dx + q[:, 2, None, None] * dy * dy)
        sigma = size + q[:, 1, None, None] * dx * dy
        same &= ~((np.abs(sigma) < 1e-4 + 1e-5 * size) | ((size > 200.0) & (sigma < 10.0)))
    assert same.mean() > 0.8
    mask, mk = t(same[..., None].astype(np.float32)), same[..., None].astype(np.float64)
    leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
    out_c, out_a = ops.rasterize_to_pixels(*(leaves[k] for k in keys), W, H, ts, t(c["offsets"], torch.int32),
                                           t(c["flatten_ids"], torch.int32), t(c["rs"]), absgrad=absgrad)
    for got, want in ((out_c, f32["render_colors"]), (out_a, f32["render_alphas"])):
        assert_close(f"pixels tile {ts} ch={channels}", n(got), want, 1e-4, 1e-5, mask=same[..., None])
    torch.autograd.backward([out_c, out_a], [t(v_c) * mask, t(v_a) * mask])
    ref = composite.rasterize_to_pixels_bwd(*args, ref_f["render_alphas"], ref_f["last_ids"], n(v_c) * mk, n(v_a) * mk,
                                            absgrad=absgrad)
    plain = np.r_[0:2, 6:120]   # the needles' own gradients are sums of large terms that cancel
    for k in keys:
        _grad_check(f"tile {ts} ch={channels} v_{k}", leaves[k].grad[:, plain], ref["v_" + k].reshape(leaves[k].shape)[:, plain])
    if absgrad:
        _grad_check(f"tile {ts} ch={channels} absgrad", leaves["means2d"].absgrad[:, plain],
                    ref["v_means2d_abs"].reshape(C, 120, 2)[:, plain])


@pytest.mark.parametrize("C,ts,channels,absgrad", [(12, 16, 30, True), (24, 16, 3, False), (24, 16, 7, True), (24, 16, 13, False), (24, 16, 20, True),
                                                   (43, 16, 4, False), (84, 16, 3, True), (60, 16, 13, True), (60, 20, 8, False), (300, 8, 4, False)])
def test_pixels_by_how_many_tiles_a_gaussian_covers(C, ts, channels, absgrad):
    """The hint that chooses how many pixels a lane draws changes no bit of an image, a background and a divided depth among
    them; every choice matches the oracle, forward and backward."""
    from oracle import composite
    from splatad_b200 import ops
    W, H = (127, 133) if C % 2 else (132, 131)
    c = _camera_case(C, 60, W, H, ts, channels, 100 * ts + channels, sigma_px=(1.0, 9.0))
    g = torch.Generator().manual_seed(7)
    bg = torch.rand(C, channels, generator=g)
    v_c, v_a = torch.randn(C, H, W, channels, generator=g), torch.randn(C, H, W, 1, generator=g)
    keys = ("means2d", "conics", "colors", "opacities", "pix_vels")
    args = [n(c[k]) for k in keys] + [n(c["rs"]), n(bg), W, H, ts, c["offsets"], c["flatten_ids"]]
    ref_f = composite.rasterize_to_pixels_fwd(*args, dtype=np.float64)
    f32 = composite.rasterize_to_pixels_fwd(*args, amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    assert same.mean() > 0.9
    mask, mk = t(same[..., None].astype(np.float32)), same[..., None].astype(np.float64)
    ref = composite.rasterize_to_pixels_bwd(*args, ref_f["render_alphas"], ref_f["last_ids"], n(v_c) * mk, n(v_a) * mk,
                                            absgrad=absgrad)
    offsets, ids = t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32)
    first = None
    for spread, count in ((0.0, 0), (2.0, 10**7), (4.5, 10**7), (6.5, 10**7), (8.0, 10**7), (12.0, 700_000), (12.0, 10**5), (20.0, 10**7)):
        ids._splatad_spread, ids._splatad_count = spread, count
        leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
        out_c, out_a = ops.rasterize_to_pixels(*(leaves[k] for k in keys), W, H, ts, offsets, ids, t(c["rs"]), backgrounds=t(bg),
                                               absgrad=absgrad)
        if first is None:
            first = out_c, out_a
            for got, want in ((out_c, f32["render_colors"]), (out_a, f32["render_alphas"])):
                assert_close(f"pixels tile {ts} ch={channels}", n(got), want, 1e-4, 1e-5, mask=same[..., None])
        assert torch.equal(out_c, first[0]) and torch.equal(out_a, first[1])
        torch.autograd.backward([out_c, out_a], [t(v_c) * mask, t(v_a) * mask])
        for k in keys:
            _grad_check(f"tile {ts} ch={channels} spread {spread} v_{k}", leaves[k].grad, ref["v_" + k].reshape(leaves[k].shape))
        if absgrad:
            _grad_check(f"tile {ts} ch={channels} spread {spread} absgrad", leaves["means2d"].absgrad,
                        ref["v_means2d_abs"].reshape(C, 60, 2))


@pytest.mark.parametrize("C,W,H,ts,channels,sigma_px,N,absgrad", [
    (30, 127, 133, 16, 3, (20.0, 90.0), 150, False), (84, 132, 131, 16, 4, (20.0, 90.0), 90, True), (30, 128, 128, 16, 1, (3.0, 60.0), 200, True),
    (84, 121, 120, 16, 2, (60.0, 400.0), 64, False), (24, 131, 129, 32, 4, (10.0, 90.0), 150, False), (110, 130, 130, 24, 3, (20.0, 90.0), 90, False),
    (30, 127, 133, 16, 7, (20.0, 90.0), 90, True), (30, 132, 131, 16, 14, (10.0, 90.0), 90, False),
    (30, 127, 133, 16, 5, (20.0, 90.0), 90, False), (24, 131, 130, 16, 7, (10.0, 90.0), 90, False), (30, 128, 131, 16, 8, (20.0, 90.0), 90, False),
    (24, 132, 129, 16, 16, (20.0, 90.0), 90, True)])
def test_runs_of_entries_that_cover_a_patch(C, W, H, ts, channels, sigma_px, N, absgrad):
    """Scenes of large Gaussians: entries that cover a patch go through without a test in the kernel for them, which the hint
    chooses - forward up to four channels, backward up to sixteen, and not where a tile's rows leave lanes over (24 pixels) -; images, alphas
    and last positions are those of the kernel without runs, bit for bit, and match the oracle, as the gradients do. Opaque
    and capped entries, needles, a flat conic and ones that cover part of a patch among them."""
    from oracle import composite
    from splatad_b200 import _lib
    c = _camera_case(C, N, W, H, ts, channels, 31 * ts + channels, sigma_px=sigma_px)
    q = c["conics"]
    q[:, 0] = torch.tensor([0.5, 0.495, 0.5])         # a needle
    q[:, 1] = torch.tensor([1e-6, 0.0, 1e-6])         # covers everything
    q[:, 2] = torch.tensor([1e-4, 0.99e-4, 1e-4])     # as narrow, but large
    c["opacities"][:, 3] = 0.9985
    c["opacities"][:, 4:9] = 0.02
    keys = ("means2d", "conics", "colors", "opacities", "pix_vels")
    args = [n(c[k]) for k in keys] + [n(c["rs"]), None, W, H, ts, c["offsets"], c["flatten_ids"]]
    want, exact = composite.rasterize_to_pixels_fwd(*args, amb_tol=1e-4), composite.rasterize_to_pixels_fwd(*args, dtype=np.float64)
    ok = ~want["ambiguous"] & (want["last_ids"] == exact["last_ids"])
    assert ok.mean() > 0.9
    g = torch.Generator().manual_seed(5)
    v_c, v_a = (torch.randn(C, H, W, k, generator=g) * torch.from_numpy(ok[..., None]) for k in (channels, 1))
    ref = composite.rasterize_to_pixels_bwd(*args, exact["render_alphas"], exact["last_ids"], n(v_c), n(v_a), absgrad=absgrad)
    lib, p = _lib.load(), _lib.ptr
    dev = {k: t(c[k]) for k in keys + ("rs",)}
    offsets, ids = t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32)
    th, tw = c["offsets"].shape[1:]
    head = (C, ids.numel(), *(p(dev[k]) for k in keys[:3]), channels, p(dev["opacities"]), p(dev["pix_vels"]), p(dev["rs"]), None, W, H, ts,
            tw, th, p(offsets), p(ids))
    cotangents, first = (v_c.to(DEV), v_a.to(DEV)), None
    for spread, count in ((0.0, 0), (100.0, 10**8)):
        image, alphas = torch.empty(C, H, W, channels, device=DEV), torch.empty(C, H, W, 1, device=DEV)
        last = torch.empty(C, H, W, dtype=torch.int32, device=DEV)
        lib.splatad_rasterize_set_spread_hint(spread, count), lib.splatad_rasterize_set_near_hint(4 * spread)
        _, (name,) = launched(lambda: _lib.call("splatad_rasterize_to_pixels_fwd", *head, p(image), p(alphas), p(last),
                                                _lib.stream_ptr(ids.device)))
        assert name.endswith(",runs") == (spread > 0 and channels <= 4 and ts != 24), name
        if first is None:
            first = image, alphas, last
            assert_close("image", n(image), want["render_colors"], 1e-4, 1e-5, mask=ok[..., None])
            assert (n(last) == want["last_ids"])[ok].all()
        for got, expect in zip((image, alphas, last), first):
            assert torch.equal(got, expect)
        v = {k: torch.zeros_like(dev[k]) for k in keys}
        v_abs = torch.zeros_like(dev["means2d"]) if absgrad else None
        lib.splatad_rasterize_set_spread_hint(spread, count), lib.splatad_rasterize_set_near_hint(4 * spread)
        _, (name,) = launched(lambda: _lib.call(
            "splatad_rasterize_to_pixels_bwd", *head, p(alphas), p(last), p(cotangents[0]), p(cotangents[1]), p(v_abs),
            *(p(v[k]) for k in ("means2d", "conics", "colors", "opacities", "pix_vels")), _lib.stream_ptr(ids.device)))
        assert name.endswith(",runs") == (spread > 0 and ts != 24), name
        for k in keys:
            _grad_check(f"spread {spread} v_{k}", v[k], ref["v_" + k].reshape(v[k].shape))
        if absgrad:
            _grad_check(f"spread {spread} absgrad", v_abs, ref["v_means2d_abs"].reshape(v_abs.shape))


def _chosen(C, W, H, ts, spread, per_tile, near, channels):
    """Names of the forward and the backward kernel that hints choose; drawn are empty lists."""
    from splatad_b200 import _lib
    lib, p = _lib.load(), _lib.ptr
    tw, th = -(-W // ts), -(-H // ts)
    offsets, ids = torch.ones(C, th, tw, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)   # empty lists
    image, alphas, one = torch.empty(C, H, W, channels, device=DEV), torch.zeros(C, H, W, 1, device=DEV), torch.zeros(32, device=DEV)
    last, rs = torch.full((C, H, W), -1, dtype=torch.int32, device=DEV), torch.zeros(C, device=DEV)
    head = (C, 1, p(one), p(one), p(one), channels, p(one), p(one), p(rs), None, W, H, ts, tw, th, p(offsets), p(ids))
    grads = [torch.zeros(32, device=DEV) for _ in range(5)]
    entries = per_tile * C * tw * th

    def both():
        lib.splatad_rasterize_set_spread_hint(spread, entries), lib.splatad_rasterize_set_near_hint(near)
        _lib.call("splatad_rasterize_to_pixels_fwd", *head, p(image), p(alphas), p(last), _lib.stream_ptr(ids.device))
        lib.splatad_rasterize_set_spread_hint(spread, entries), lib.splatad_rasterize_set_near_hint(near)
        _lib.call("splatad_rasterize_to_pixels_bwd", *head, p(alphas), p(last), p(image), p(alphas), None, *(p(g) for g in grads),
                  _lib.stream_ptr(ids.device))

    return launched(both)[1]


@pytest.mark.parametrize("W,H,channels,runs", [(960, 400, 8, False), (960, 400, 4, True), (960, 400, 14, True), (800, 496, 8, True), (800, 496, 5, True),
                                              (800, 496, 17, False), (1200, 296, 8, False)])
def test_backward_runs_by_channels(W, H, channels, runs):
    """Up to sixteen channels; five to eight not where the warps without runs just fit at once."""
    assert _chosen(1, W, H, 16, 20.0, 1800, 900, channels)[1].endswith(",runs") == runs


@pytest.mark.parametrize("C,W,H,ts,spread,per_tile,near,forward,backward", [
    (2, 640, 360, 16, 68.0, 573, 900, False, True), (2, 640, 360, 16, 38.0, 1400, 900, True, True), (1, 1280, 720, 16, 59.0, 596, 900, False, True),
    (1, 1280, 720, 16, 23.0, 2296, 900, True, True), (2, 1280, 720, 16, 81.0, 162, 900, False, True), (2, 1280, 720, 16, 79.0, 316, 900, True, True),
    (3, 1440, 430, 16, 43.0, 372, 900, False, True), (4, 640, 800, 16, 31.0, 439, 900, True, True), (1, 1920, 1080, 16, 27.0, 1171, 900, True, True),
    (1, 1920, 1080, 16, 16.0, 682, 900, False, False), (1, 640, 360, 16, 79.0, 3643, 900, False, True), (1, 480, 270, 16, 79.0, 9000, 900, False, False),
    (1, 1280, 720, 24, 59.0, 5000, 900, False, False), (1, 1280, 720, 32, 20.0, 5000, 300, True, True), (1, 1920, 1080, 16, 27.0, 1171, 349, False, True),
    (1, 1920, 1080, 16, 27.0, 1171, 351, True, True), (1, 1920, 1080, 16, 37.0, 9673, 40, False, False), (1, 1920, 1080, 16, 27.0, 1171, 176, False, True),
    (1, 1920, 1080, 16, 27.0, 1171, 0, False, False)])
def test_runs_are_for_dense_lists_of_large_gaussians(C, W, H, ts, spread, per_tile, near, forward, backward):
    """Which camera kernels the hints choose, on both sides of each line: near Gaussians that are small or of no known size, sparse lists, few
    tiles, rows that leave lanes over."""
    names = _chosen(C, W, H, ts, spread, per_tile, near, 3)
    assert [k.endswith("_kernel/8,runs") for k in names] == [forward, backward], names


def test_runs_of_thousands_of_faint_entries():
    """Every entry covers every patch with an alpha just above 1/255, so that some 2250 of them go by before a transmittance comes
    near the limit, the longest sum that the bound of the transmittances is ever taken over: each pixel stops where it does
    without runs, and the images are the same bit for bit."""
    from splatad_b200 import _lib
    C, W, H, ts, N = 2, 480, 480, 16, 2600
    g = torch.Generator().manual_seed(9)
    tw, th = W // ts, H // ts
    means2d, colors = torch.rand(C, N, 2, generator=g) * torch.tensor([W, H]), torch.rand(C, N, 3, generator=g)
    conics = torch.tensor([2e-8, 0.0, 2e-8]).expand(C, N, 3).contiguous()
    opacities = 1.005 / 255 * (1 + 0.08 * torch.rand(C, N, generator=g))
    dev = [x.to(DEV) for x in (means2d, conics, colors, opacities, torch.zeros(C, N, 2), torch.zeros(C))]
    offsets = (torch.arange(C * tw * th, dtype=torch.int32) * N).to(DEV)
    ids = torch.arange(C * N, dtype=torch.int32).view(C, 1, N).expand(C, tw * th, N).contiguous().to(DEV)
    lib, p, results = _lib.load(), _lib.ptr, []
    for hint, runs in (((0.0, 0), False), ((100.0, 10**8), True)):
        image, alphas = torch.empty(C, H, W, 3, device=DEV), torch.empty(C, H, W, 1, device=DEV)
        last = torch.empty(C, H, W, dtype=torch.int32, device=DEV)
        lib.splatad_rasterize_set_spread_hint(*hint), lib.splatad_rasterize_set_near_hint(4 * hint[0])
        _, (name,) = launched(lambda: _lib.call(
            "splatad_rasterize_to_pixels_fwd", C, ids.numel(), *(p(x) for x in dev[:3]), 3, *(p(x) for x in dev[3:]), None, W, H, ts, tw, th,
            p(offsets), p(ids), p(image), p(alphas), p(last), _lib.stream_ptr(ids.device)))
        assert name.endswith(",runs") == runs, name
        results.append((image, alphas, last))
    for a, b in zip(*results):
        assert torch.equal(a, b)
    at = results[0][2].view(C, th, ts, tw, ts) % N   # (each tile's list has the N entries of its camera)
    assert 2000 < int(at.min()) and int(at.max()) < N - 100


@pytest.mark.parametrize("channels,absgrad", [(3, False), (8, False), (8, True), (14, False)])
@pytest.mark.parametrize("what", ["colors", "means2d", "conics", "opacities", "flat", "cotangent"])
def test_runs_with_values_that_are_not_finite(what, channels, absgrad):
    """The kernels with runs (above four channels the backward ones) and those without them agree on the pixels that a value which is
    not finite reaches, on the Gaussians that get such a gradient, and on all others."""
    from splatad_b200 import _lib
    C, W, H, ts, N = 30, 128, 127, 16, 90
    c = _camera_case(C, N, W, H, ts, channels, 77, sigma_px=(15.0, 80.0))
    if what == "flat": c["conics"][:, 5] = torch.tensor([1e-37, 0.0, 1e-37])
    elif what != "cotangent":
        c[what][:, 5], c[what][::2, 11] = float("nan"), float("inf")
    g = torch.Generator().manual_seed(2)
    v_c, v_a = torch.randn(C, H, W, channels, generator=g), torch.randn(C, H, W, 1, generator=g)
    if what == "cotangent": v_c[::3, 40, 50, 1], v_a[1, 3, 3] = float("nan"), float("inf")
    lib, p = _lib.load(), _lib.ptr
    keys = ("means2d", "conics", "colors", "opacities", "pix_vels")
    dev = {k: t(c[k]) for k in keys + ("rs",)}
    offsets, ids, v_c, v_a = t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), t(v_c), t(v_a)
    th, tw = c["offsets"].shape[1:]
    head = (C, ids.numel(), *(p(dev[k]) for k in keys[:3]), channels, p(dev["opacities"]), p(dev["pix_vels"]), p(dev["rs"]), None, W, H, ts,
            tw, th, p(offsets), p(ids))
    results, hints = [], ((0.0, 0), (100.0, 10**8))
    for hint in hints:
        image, alphas = torch.empty(C, H, W, channels, device=DEV), torch.empty(C, H, W, 1, device=DEV)
        last = torch.empty(C, H, W, dtype=torch.int32, device=DEV)
        lib.splatad_rasterize_set_spread_hint(*hint), lib.splatad_rasterize_set_near_hint(4 * hint[0])
        _lib.call("splatad_rasterize_to_pixels_fwd", *head, p(image), p(alphas), p(last), _lib.stream_ptr(ids.device))
        results.append((image, alphas, last))
    (image, alphas, last), (image_r, alphas_r, last_r) = results
    same = ((last & 0x7FFFFFFF) == (last_r & 0x7FFFFFFF))[..., None]
    v_c, v_a, gradients = torch.where(same, v_c, 0.0), torch.where(same, v_a, 0.0), []
    for hint, (_, alphas_h, last_h) in zip(hints, results):
        grads = {k: torch.zeros_like(dev[k]) for k in keys}
        if absgrad:
            grads["absgrad"] = torch.zeros_like(dev["means2d"])
        lib.splatad_rasterize_set_spread_hint(*hint), lib.splatad_rasterize_set_near_hint(4 * hint[0])
        _, (name,) = launched(lambda: _lib.call(
            "splatad_rasterize_to_pixels_bwd", *head, p(alphas_h), p(last_h), p(v_c), p(v_a), p(grads.get("absgrad")),
            *(p(grads[k]) for k in ("means2d", "conics", "colors", "opacities", "pix_vels")), _lib.stream_ptr(ids.device)))
        assert name.endswith(",runs") == (hint[1] > 0), name
        gradients.append(grads)
    v, v_r = gradients
    # pixels are worked out again patch by patch, and patches differ in size: a rounding, and a decision in a few thousand, may differ
    assert_close("alphas", n(alphas_r), n(alphas), 1e-4, 1e-5, max_bad_frac=1e-3)
    assert same.float().mean() > 0.999
    assert (image.isfinite() == image_r.isfinite()).float().mean() > 0.9999
    both = image.isfinite() & image_r.isfinite()
    assert_close("image", n(image_r), n(image), 1e-4, 1e-5, mask=n(both).astype(bool), max_bad_frac=1e-3)
    for k in v:
        assert (v[k].isfinite() == v_r[k].isfinite()).float().mean() > 0.999, k
        both = v[k].isfinite() & v_r[k].isfinite()
        _grad_check(k, torch.where(both, v_r[k], 0.0), n(torch.where(both, v[k], 0.0)), rel=5e-3)


@pytest.mark.parametrize("C,channels", [(24, 3), (43, 4), (84, 2), (24, 13), (12, 30)])
def test_divided_depth_of_many_tiles(C, channels):
    """The last channel divided by the alpha inside the kernels, forward and backward, against the same division behind them,
    for every choice of pixels per lane."""
    from splatad_b200 import _lib, ops
    W, H, ts = 132, 131, 16
    c = _camera_case(C, 60, W, H, ts, channels, 9 * channels, sigma_px=(1.0, 9.0))
    keys = ("means2d", "conics", "colors", "opacities", "pix_vels")
    dev = {k: t(c[k]) for k in keys}
    bg, rs = torch.zeros(C, channels, device=DEV), t(c["rs"])
    bg[:, :-1] = 0.3
    offsets, ids = t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32)
    g = torch.Generator(device=DEV).manual_seed(8)
    v_c, v_a = torch.randn(C, H, W, channels, generator=g, device=DEV), torch.randn(C, H, W, 1, generator=g, device=DEV)
    leaves = {k: v.clone().requires_grad_(True) for k, v in dev.items()}
    out_c, out_a = ops.rasterize_to_pixels(*(leaves[k] for k in keys), W, H, ts, offsets, ids, rs, backgrounds=bg)
    want = torch.cat([out_c[..., :-1], out_c[..., -1:] / out_a.clamp(min=1e-10)], -1)
    torch.autograd.backward([want, out_a], [v_c, v_a])
    lib, p = _lib.load(), _lib.ptr
    th, tw = c["offsets"].shape[1:]
    for spread in (0.0, 2.0, 6.5, 20.0):
        image, alphas = torch.empty(C, H, W, channels, device=DEV), torch.empty(C, H, W, 1, device=DEV)
        last, depths = torch.empty(C, H, W, dtype=torch.int32, device=DEV), torch.empty(C, H, W, device=DEV)
        head = (C, ids.numel(), p(dev["means2d"]), p(dev["conics"]), p(dev["colors"]), channels, p(dev["opacities"]), p(dev["pix_vels"]),
                p(rs), p(bg), W, H, ts, tw, th, p(offsets), p(ids))
        lib.splatad_rasterize_set_spread_hint(spread, 10**7)
        _lib.call("splatad_rasterize_expected_to_pixels_fwd", *head, 1, p(image), p(alphas), p(last), p(depths), _lib.stream_ptr(ids.device))
        assert_close(f"depth ch={channels} spread {spread}", n(image), n(want), 1e-6, 1e-7)
        assert torch.equal(alphas, out_a) and torch.equal(depths, image[..., -1])
        v = [torch.zeros_like(dev[k]) for k in ("means2d", "conics", "colors", "opacities", "pix_vels")]
        lib.splatad_rasterize_set_spread_hint(spread, 10**7)
        _lib.call("splatad_rasterize_expected_to_pixels_bwd", *head, p(depths), p(alphas), p(last), p(v_c), p(v_a), None, *(p(x) for x in v),
                  _lib.stream_ptr(ids.device))
        for k, got in zip(keys, v):
            _grad_check(f"depth ch={channels} spread {spread} v_{k}", got, n(leaves[k].grad))


@pytest.mark.parametrize("tw,th,H,W,channels,asum,absgrad", [(32, 8, 20, 130, 3, True, True), (8, 4, 9, 100, 17, False, False),
                                                             (5, 3, 10, 64, 9, True, False), (64, 16, 40, 96, 16, False, True),
                                                             (1, 1, 6, 40, 2, True, False), (32, 8, 130, 1024, 5, True, False),
                                                             (8, 8, 17, 70, 32, False, False)])
def test_points_in_patches(tw, th, H, W, channels, asum, absgrad):
    """Patches of 8 x 4 and 8 x 8 points, tiles that cannot be cut into them, scans that end inside a
    patch, patches without a single return, one and several CTAs per tile, few tiles and many:
    forward and backward against the oracle."""
    from oracle import composite
    from splatad_b200 import ops
    c = _lidar_case(1, 1500, H, W, tw, th, channels, 100 * tw + channels)
    c["pts"][0, : min(th, H), : min(tw, W), 2] = 0.0
    g = torch.Generator().manual_seed(4)
    v_c, v_a, v_s = (torch.randn(1, H, W, k, generator=g) for k in (channels, 1, 1))
    keys = ("means2d", "conics", "feats", "opacities", "pix_vels", "dcomp")
    args = [n(c[k]) for k in keys] + [None, n(c["pts"]), W, H, tw, th, c["offsets"], c["flatten_ids"], asum, 0.5]
    ref_f = composite.rasterize_to_points_fwd(*args, dtype=np.float64)
    f32 = composite.rasterize_to_points_fwd(*args, amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    assert same.mean() > 0.9
    mask, mk = t(same[..., None].astype(np.float32)), same[..., None].astype(np.float64)
    leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
    out_c, out_a, out_s, out_m = ops.rasterize_to_points(
        *(leaves[k] for k in keys), t(c["pts"]), W, H, tw, th, t(c["offsets"], torch.int32),
        t(c["flatten_ids"], torch.int32), asum, 0.5, absgrad=absgrad)
    _check_fwd(f"points tile {tw}x{th} ch={channels}", n(out_c), n(out_a), f32, depth_channel=channels - 1)
    cot = [t(v_c) * mask, t(v_a) * mask] + ([t(v_s) * mask] if asum else [])
    torch.autograd.backward([out_c, out_a] + ([out_s] if asum else []), cot)
    ref = composite.rasterize_to_points_bwd(*args, ref_f["render_alphas"], ref_f["last_ids"], n(v_c) * mk, n(v_a) * mk,
                                            (n(v_s) * mk) if asum else None, absgrad=absgrad)
    names = ("v_means2d", "v_conics", "v_colors", "v_opacities", "v_pix_vels", "v_depth_comps")
    for k, name in zip(keys, names):
        _grad_check(f"tile {tw}x{th} ch={channels} {name}", leaves[k].grad, ref[name])
    if absgrad:
        _grad_check(f"tile {tw}x{th} ch={channels} absgrad", leaves["means2d"].absgrad, ref["v_means2d_abs"])


@pytest.mark.parametrize("C,N,channels,shared", [(2, 400, 5, True), (2, 65_000, 5, False), (2, 500, 13, True), (2, 39_000, 13, False),
                                                 (2, 400, 24, False)])
def test_points_of_sparse_and_dense_scenes(C, N, channels, shared):
    """Scans of 1184 to 1479 patches share a patch between the warps of a block where the scene is sparse. Either way gives the
    oracle's features, and the same transmittances bit for bit as without the hint."""
    from oracle import composite
    from splatad_b200 import _lib, ops
    H, W, tw, th = 64, 320, 32, 8                      # 1280 patches
    c = _lidar_case(C, N, H, W, tw, th, channels, 3 * N + channels)
    assert (C * N < 1280 * (100 if channels <= 8 else 60) and channels <= 20) == shared
    keys = ("means2d", "conics", "feats", "opacities", "pix_vels", "dcomp")
    ref = composite.rasterize_to_points_fwd(*(n(c[k]) for k in keys), None, n(c["pts"]), W, H, tw, th, c["offsets"], c["flatten_ids"],
                                            True, 0.5)
    dev = [t(c[k]) for k in keys]
    offsets, ids, pts = t(c["offsets"], torch.int32), t(c["flatten_ids"], torch.int32), t(c["pts"])
    out_c, out_a, out_s, out_m = ops.rasterize_to_points(*dev, pts, W, H, tw, th, offsets, ids, True, 0.5)
    sure = ~ref["ambiguous"][..., None]
    assert_close("features", n(out_c), ref["render_colors"], 2e-4, 2e-5, mask=sure)
    assert_close("alphas", n(out_a), ref["render_alphas"], 2e-4, 2e-5, mask=sure)
    # without the hint: one warp to a patch
    p, f = _lib.ptr, torch.float32
    image, alphas, sums, medians = (torch.empty(C, H, W, k, device=DEV, dtype=f) for k in (channels, 1, 1, 1))
    last = torch.empty(C, H, W, dtype=torch.int32, device=DEV)
    _lib.call("splatad_rasterize_to_points_fwd", C, ids.numel(), p(dev[0]), p(dev[1]), p(dev[2]), None, channels, p(dev[3]), p(dev[4]), p(dev[5]),
              None, p(pts), W, H, tw, th, offsets.shape[2], offsets.shape[1], 1, 0.5, p(offsets), p(ids), channels - 1, p(image), p(alphas), p(sums),
              p(last), p(medians), _lib.stream_ptr(ids.device))
    assert torch.equal(alphas, out_a)
    assert_close("medians", n(medians), n(out_m), 1e-5, 1e-6)  # of the same entry, its range term rounded in another order
    assert_close("features", n(image), n(out_c), 1e-5, 1e-6)   # sums of eight warps added in order, 32-bit
    assert torch.equal(image, out_c) or shared


@pytest.mark.parametrize("C,H,W,channels", [(1, 16, 256, 3), (1, 32, 300, 9), (6, 64, 512, 5), (6, 64, 512, 18)])
def test_points_with_needles_and_the_seam(C, H, W, channels):
    """Entries whose alphas or angles need care beside those that do not - needles on either side of the line, a conic that
    is not positive definite, opacities above the cap, means on both sides of the half turn - where the warps of a CTA
    share a patch and where they do not, forward and backward against the oracle."""
    from oracle import composite
    from splatad_b200 import ops
    N, tw, th = 400, 32, 8
    c = _lidar_case(C, N, H, W, tw, th, channels, 77 * H + channels)
    c["opacities"][:, ::11] = 0.9995
    for k, rho in enumerate((0.999, 0.99999, 0.9999999, 1.5)):   # 1 - rho^2 against 1e-5
        a, b = c["conics"][:, 2 + k, 0], c["conics"][:, 2 + k, 2]
        c["conics"][:, 2 + k, 1] = rho * torch.sqrt(a * b)
    g = torch.Generator().manual_seed(4)
    v_c, v_a, v_s = (torch.randn(C, H, W, k, generator=g) for k in (channels, 1, 1))
    keys = ("means2d", "conics", "feats", "opacities", "pix_vels", "dcomp")
    args = [n(c[k]) for k in keys] + [None, n(c["pts"]), W, H, tw, th, c["offsets"], c["flatten_ids"], True, 0.5]
    ref_f = composite.rasterize_to_points_fwd(*args, dtype=np.float64)
    f32 = composite.rasterize_to_points_fwd(*args, amb_tol=1e-4)
    same = (f32["last_ids"] == ref_f["last_ids"]) & ~f32["ambiguous"]
    # the sign and the size of a form that nearly vanishes or is negative somewhere hang on the last bits
    pts = n(c["pts"]).astype(np.float64)
    turn = lambda d: (d + 180.0) % 360.0 - 180.0   # noqa: E731
    for k in range(2, 6):
        m, v, q = (n(c[key])[:, k].astype(np.float64)[:, None, None] for key in ("means2d", "pix_vels", "conics"))
        dx, dy = turn(m[..., 0] + pts[..., 3] * v[..., 0] - pts[..., 0]), m[..., 1] + pts[..., 3] * v[..., 1] - pts[..., 1]
        size = 0.5 * (q[..., 0] * dx * dx + q[..., 2] * dy * dy)
        sigma = size + q[..., 1] * dx * dy
        same &= ~((sigma < 12.0) & ((size > 20.0) | (np.abs(sigma) < 1e-3)))
    assert same.mean() > 0.6   # four needles and the one with two signs reach a third of the smallest scan
    mask, mk = t(same[..., None].astype(np.float32)), same[..., None].astype(np.float64)
    leaves = {k: t(c[k]).requires_grad_(True) for k in keys}
    out_c, out_a, out_s, _ = ops.rasterize_to_points(*(leaves[k] for k in keys), t(c["pts"]), W, H, tw, th, t(c["offsets"], torch.int32),
                                                     t(c["flatten_ids"], torch.int32), True, 0.5)
    for got, want in ((out_c, f32["render_colors"]), (out_a, f32["render_alphas"])):
        assert_close(f"points {H}x{W} ch={channels}", n(got), want, 2e-4, 2e-5, mask=same[..., None])
    torch.autograd.backward([out_c, out_a, out_s], [t(v_c) * mask, t(v_a) * mask, t(v_s) * mask])
    ref = composite.rasterize_to_points_bwd(*args, ref_f["render_alphas"], ref_f["last_ids"], n(v_c) * mk, n(v_a) * mk, n(v_s) * mk)
    plain = np.r_[0:2, 6:N]   # the needles' own gradients are sums of large terms that cancel
    names = ("v_means2d", "v_conics", "v_colors", "v_opacities", "v_pix_vels", "v_depth_comps")
    for k, name in zip(keys, names):
        _grad_check(f"points {H}x{W} ch={channels} {name}", leaves[k].grad[:, plain], ref[name].reshape(leaves[k].shape)[:, plain])
