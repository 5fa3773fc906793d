"""Frames through the native host side (``csrc/host/frames.cpp``): from the second frame of a shape on, one call
enqueues the frame and puts its own two nodes into the autograd graph. Whatever it takes, its images, lists,
gradients and refusals are those of the individual ops."""

import pytest
import torch

from gpu_util import DEV, launched

pytestmark = pytest.mark.gpu


def _to_gpu(cfg):
    return {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in cfg.items()}


def _forget():
    """No frame has a predecessor: the next one is rendered by the individual ops."""
    from splatad_b200 import ops
    for hint in (ops._isect_count_hint, ops._packed_nnz_hint, ops._depth_range_hint, ops._depth_sort_mode):
        hint.clear()


@pytest.mark.parametrize("packed", [False, True])
def test_a_frame_reports_how_many_tiles_its_gaussians_cover(packed):
    """List entries per Gaussian that the lists hold: from the ops in a first frame, from the plan's own words in the next
    ones. It goes with the lists and chooses how the next frame is split, which changes no bit of its image."""
    import splatad_b200
    from splatad_b200 import ops, scenes
    g = _to_gpu(scenes.config1(N=20_011, packed=packed))
    _forget()
    first = None
    for hint in (None, None, 1.0, 6.0, 50.0):
        if hint is None and first is None:
            ops._spread_hint.clear()
        elif hint is not None:
            ops._spread_hint[next(iter(ops._spread_hint))] = hint
        image, alpha, meta = splatad_b200.rasterization(**g)
        want = meta["flatten_ids"].numel() / int((meta["tiles_per_gauss"] > 0).sum())
        assert list(ops._spread_hint.values()) == [pytest.approx(want)] and want > 1.0
        assert meta["flatten_ids"]._splatad_spread == pytest.approx(want)
        first = first or (image, alpha)
        assert torch.equal(image, first[0]) and torch.equal(alpha, first[1])


@pytest.mark.parametrize("packed,pose", [(False, False), (True, False), (False, True)])
def test_a_frame_is_split_by_its_own_counts(packed, pose):
    """Scenes of one shape in turn - Gaussians that are large where they are near, small ones, and ones that all cover 36 tiles or so, whose
    lists are as long and whose patches few of them cover: each takes the compositing kernels it takes by itself, and only the first those
    with runs, forward and backward, in native frames and (with a pose that is optimised) by the ops."""
    import splatad_b200
    from splatad_b200 import scenes
    g = _to_gpu(scenes.config1(N=150_011, packed=packed))
    if pose:
        g["viewmats"] = g["viewmats"].clone().requires_grad_(True)
    even = g["means"][:, 2:].clamp(min=0.3) * (12.0 / 1200.0)
    scales = {"large": g["scales"] * 1.5, "small": g["scales"] * 0.25, "even": even.expand(-1, 3) * 1.0}

    def step(which):
        leaf = scales[which].clone().requires_grad_(True)
        image, _, _ = splatad_b200.rasterization(**{**g, "scales": leaf})
        image.sum().backward()

    def kernels(which):
        names = [k for k in launched(lambda: step(which))[1] if k.startswith("rasterize_to_pixels")]
        return names[-2:]   # a count that outgrows its room renders the frame twice

    alone = {}
    for which in scales:
        _forget()
        for _ in range(3):
            alone[which] = kernels(which)
    assert all(k.endswith(",runs") for k in alone["large"])
    assert not any(k.endswith(",runs") for which in ("small", "even") for k in alone[which])
    for which in ("large", "small", "large", "even", "small", "small", "even", "large"):
        assert kernels(which) == alone[which], which


@pytest.mark.parametrize("kind", ["lidar", "camera"])
def test_a_frame_that_sees_nothing_has_zero_gradients(kind):
    import splatad_b200
    from splatad_b200 import scenes
    if kind == "lidar":
        g = _to_gpu(scenes.config2(N=20_011))
        render, away = splatad_b200.lidar_rasterization, torch.tensor([0.0, 0.0, 1e4], device=DEV)
    else:
        g = _to_gpu(scenes.config1(N=20_011, packed=False))
        render, away = splatad_b200.rasterization, torch.tensor([0.0, 0.0, -1e4], device=DEV)
    names = ("means", "quats", "scales", "opacities", "lidar_features" if kind == "lidar" else "colors")
    _forget()
    render(**g)                                        # its counts size the next frame of the shape
    leaves = {k: g[k].clone().requires_grad_(True) for k in names}
    *images, meta = render(**{**g, **leaves, "means": leaves["means"] + away}, absgrad=True)
    assert meta["flatten_ids"].numel() == 0 and float(images[1].detach().abs().max()) == 0.0
    meta["means2d"].retain_grad()
    sum(i.sum() for i in images).backward()
    for k in names:
        assert leaves[k].grad is not None and float(leaves[k].grad.abs().max()) == 0.0, k
    assert float(meta["means2d"].grad.abs().max()) == 0.0 and float(meta["means2d"].absgrad.abs().max()) == 0.0


@pytest.mark.parametrize("kind,name", [("lidar", "velocities"), ("lidar", "linear_velocity"), ("lidar", "raster_pts"),
                                       ("camera", "velocities"), ("camera", "Ks"), ("camera", "rolling_shutter_time")])
def test_a_tensor_without_a_gradient_of_its_own_keeps_the_frame_in_the_graph(kind, name):
    """The ops take it as an input of a node and give it no gradient; so does a frame's second call."""
    import splatad_b200
    from splatad_b200 import scenes
    g = _to_gpu(scenes.config2(N=20_011) if kind == "lidar" else scenes.config1(N=20_011))
    render = splatad_b200.lidar_rasterization if kind == "lidar" else splatad_b200.rasterization
    if g.get(name) is None:
        assert name == "velocities"
        g[name] = torch.zeros_like(g["means"])
    g[name] = g[name].clone().requires_grad_(True)
    _forget()
    for _ in range(2):
        images = render(**g)
        assert images[0].requires_grad
        images[0].sum().backward()
        assert g[name].grad is None


@pytest.mark.parametrize("rasterize_mode", ["classic", "antialiased"])
@pytest.mark.parametrize("name", ["opacities", "colors"])
def test_what_the_ops_gather_may_be_edited_before_the_backward_pass(name, rasterize_mode):
    import splatad_b200
    from splatad_b200 import scenes
    g = _to_gpu(scenes.config1(N=20_011))
    g.update(sh_degree=None, colors=torch.rand(20_011, 3, device=DEV), rasterize_mode=rasterize_mode)
    _forget()
    grads = []
    for edit in (False, False, True):        # by the ops, by the native frame, and edited behind its back
        leaves = {k: g[k].clone().requires_grad_(True) for k in ("means", "scales")}
        values = g[name].clone()
        image, alphas, _ = splatad_b200.rasterization(**{**g, **leaves, name: values})
        if edit:
            values.mul_(0.5)
        (image.square().mean() + alphas.mean()).backward()
        grads.append([v.grad for v in leaves.values()])
    for a, b, c in zip(*grads):              # sums in another order (atomics): 1e-4 from run to run
        assert float((b - a).norm()) <= 5e-4 * float(a.norm())
        assert float((c - a).norm()) <= 5e-4 * float(a.norm())


@pytest.mark.parametrize("kind", ["lidar", "camera"])
def test_forward_mode_and_transforms_are_refused_as_by_the_ops(kind):
    import splatad_b200
    import torch.autograd.forward_ad as forward_ad
    from splatad_b200 import scenes
    g = _to_gpu(scenes.config2(N=20_011) if kind == "lidar" else scenes.config1(N=20_011))
    render = splatad_b200.lidar_rasterization if kind == "lidar" else splatad_b200.rasterization
    _forget()
    render(**g)                              # from here on frames of this shape are native ones
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(g["means"], torch.ones_like(g["means"]))
        with pytest.raises(NotImplementedError):
            render(**dict(g, means=dual))
    with pytest.raises(RuntimeError, match="setup_context"):
        torch.func.grad(lambda means: render(**dict(g, means=means))[0].sum())(g["means"])


def test_sensors_that_stand_still_on_several_streams():
    """More sensors on a second stream while frames of the first are in flight, a release in between: the zeros
    a frame reads are its stream's own."""
    import splatad_b200
    from splatad_b200 import _lib, scenes
    g = _to_gpu(scenes.config1(N=20_011))
    for k in ("linear_velocity", "angular_velocity", "rolling_shutter_time"):
        g[k] = None
    many = dict(g, viewmats=g["viewmats"].repeat(30, 1, 1), Ks=g["Ks"].repeat(30, 1, 1), width=160, height=90)
    _forget()
    want, want_many = splatad_b200.rasterization(**g)[0], splatad_b200.rasterization(**many)[0]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for i in range(6):
        frames = []
        for stream in streams:
            with torch.cuda.stream(stream):
                frames.append((splatad_b200.rasterization(**g)[0], splatad_b200.rasterization(**many)[0]))
                torch.full((4096,), 7.0, device=DEV)     # takes whatever memory has been given back
        torch.cuda.synchronize()
        for one, rig in frames:
            assert torch.equal(one, want) and torch.equal(rig, want_many)
        if i == 2:
            _lib.release_workspaces()


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("render_mode", ["RGB", "RGB+D", "RGB+ED", "ED"])
def test_a_render_may_be_edited_in_place(render_mode, packed):
    import splatad_b200
    from splatad_b200 import scenes
    g = _to_gpu(scenes.config1(N=20_011, packed=packed))
    g["render_mode"] = render_mode
    _forget()
    grads = []
    for edit in (False, False, True):        # by the ops, by the native frame, and edited
        leaves = {k: g[k].clone().requires_grad_(True) for k in ("means", "opacities")}
        image, alphas, _ = splatad_b200.rasterization(**{**g, **leaves})
        if edit:
            image.mul_(2.0)
        (image.square().mean() * (0.25 if edit else 1.0) + alphas.mean()).backward()
        grads.append([v.grad for v in leaves.values()])
    for a, b, c in zip(*grads):              # sums in another order (atomics): 1e-4 from run to run
        assert float((b - a).norm()) <= 5e-4 * float(a.norm())
        assert float((c - a).norm()) <= 5e-4 * float(a.norm())


def _twice(monkeypatch, name, render, kw, leaves, cotangents):
    """Images, meta and gradients of one call by the ops and one that the native function took."""
    from splatad_b200 import rendering
    native = getattr(rendering, name)
    taken = []
    monkeypatch.setattr(rendering, name, lambda *a: taken.append(native(*a)) or taken[-1])
    _forget()
    out = []
    for _ in range(2):
        params = {k: kw[k].clone().requires_grad_(True) for k in leaves}
        *images, meta = render(**{**kw, **params})
        meta["means2d"].retain_grad()
        given = [(i, w) for i, w in zip(images, cotangents(images)) if i is not None and w is not None]
        torch.autograd.backward([i for i, _ in given], [w for _, w in given])
        grads = {k: v.grad for k, v in params.items()}
        grads["means2d"], grads["absgrad"] = meta["means2d"].grad, getattr(meta["means2d"], "absgrad", None)
        out.append(([None if i is None else i.detach() for i in images], meta, grads))
    assert taken[0] is None and taken[1] is not None
    (images, meta, grads), (images2, meta2, grads2) = out
    assert set(meta) == set(meta2)
    for k, a in meta.items():
        b = meta2[k]
        if not isinstance(a, torch.Tensor):
            assert a == b, k
        elif a.dtype.is_floating_point:
            assert a.shape == b.shape and torch.allclose(a, b, rtol=1e-6, atol=1e-6), k
        else:
            assert torch.equal(a, b), k
    for a, b in zip(images, images2):
        assert (a is None) == (b is None)
        if a is not None:      # a product or a division in one kernel or two: a rounding
            assert a.shape == b.shape and float((a - b).norm()) <= 1e-6 * float(a.norm())
    for k, a in grads.items():
        b = grads2[k]
        assert (a is None) == (b is None), k
        if a is not None:      # sums in another order (atomics): 1e-4 from run to run
            assert a.shape == b.shape and float((a - b).norm()) <= 5e-4 * float(a.norm()), k


def _all_of(images):
    g = torch.Generator(device=DEV).manual_seed(1)
    return [None if i is None else torch.randn(i.shape, generator=g, device=DEV) / i.numel() for i in images]


@pytest.mark.parametrize("C,packed,colors,mode,options", [
    (1, False, "plain", "RGB", {}),
    (1, False, "plain", "RGB+D", dict(absgrad=True)),
    (1, False, "plain", "RGB+ED", dict(rasterize_mode="antialiased")),
    (1, False, "sh", "RGB+ED", dict(backgrounds=True)),
    (1, False, "sh", "D", {}),
    (1, False, "plain", "ED", dict(backgrounds=True)),
    (1, True, "plain", "RGB", dict(backgrounds=True)),
    (1, True, "plain", "RGB+ED", dict(absgrad=True)),
    (1, True, "sh", "RGB+D", dict(rasterize_mode="antialiased", absgrad=True)),
    (1, True, "sh", "ED", {}),
    (3, False, "plain", "RGB", dict(absgrad=True)),
    (3, False, "per camera", "RGB+D", dict(backgrounds=True)),
    (3, False, "per camera sh", "RGB+ED", dict(rasterize_mode="antialiased")),
    (3, True, "per camera", "RGB+ED", dict(backgrounds=True, rasterize_mode="antialiased")),
    (3, True, "per camera sh", "RGB", {}),
    (3, True, "sh", "RGB+ED", dict(absgrad=True, backgrounds=True)),
])
@pytest.mark.parametrize("cotangents", ["all", "image only", "alpha only"])
def test_native_camera_frames_are_those_of_the_ops(C, packed, colors, mode, options, cotangents, monkeypatch):
    import splatad_b200
    from splatad_b200 import scenes
    N = 8_009
    kw = _to_gpu(scenes.config1(N=N, packed=packed))
    g = torch.Generator(device=DEV).manual_seed(C)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEV)   # noqa: E731
    kw.update(width=333, height=211, render_mode=mode, scales=kw["scales"] * 2.0, **options)
    kw["Ks"] = torch.tensor([[[210.0, 0.0, 166.0], [0.0, 210.0, 105.0], [0.0, 0.0, 1.0]]], device=DEV).repeat(C, 1, 1)
    if C > 1:
        kw["viewmats"] = kw["viewmats"].repeat(C, 1, 1)
        kw["viewmats"][:, 0, 3] = torch.arange(C, device=DEV) * 2.0
        for k in ("linear_velocity", "angular_velocity"):
            kw[k] = kw[k].repeat(C, 1)
        kw["rolling_shutter_time"] = kw["rolling_shutter_time"].repeat(C)
    if "sh" not in colors:
        kw.update(sh_degree=None, colors=rand(C, N, 5) if "per camera" in colors else rand(N, 5))
    elif "per camera" in colors:
        kw["colors"] = (rand(C, N, 16, 3) - 0.5) * 0.6
    if options.get("backgrounds"):
        kw["backgrounds"] = rand(C, 3 if "sh" in colors else 5)
    wanted = {"all": _all_of, "image only": lambda i: [_all_of(i)[0], None], "alpha only": lambda i: [None, _all_of(i)[1]]}[cotangents]
    leaves = ("means", "quats", "scales", "opacities") + (() if mode in ("D", "ED") else ("colors",))
    if cotangents == "alpha only":
        leaves = tuple(k for k in leaves if k != "colors")
    _twice(monkeypatch, "_native_camera_frame", splatad_b200.rasterization, kw, leaves, wanted)


@pytest.mark.parametrize("C,features,options", [
    (1, 1, {}), (1, 7, dict(absgrad=True)), (1, 16, dict(rasterize_mode="antialiased")), (1, 4, dict(compute_alpha_sum_until_points=False)),
    (2, 4, dict(absgrad=True)), (2, 16, dict(rasterize_mode="antialiased")),
])
@pytest.mark.parametrize("cotangents", ["all", "image only", "alpha only", "alpha sum only"])
def test_native_lidar_frames_are_those_of_the_ops(C, features, options, cotangents, monkeypatch):
    import splatad_b200
    from splatad_b200 import scenes
    at = ("all", "image only", "alpha only", "alpha sum only").index(cotangents) - 1
    if at == 2 and options.get("compute_alpha_sum_until_points") is False:
        pytest.skip("no alpha sum")
    N = 15_013
    kw = _to_gpu(scenes.config2(N=N, width=600))
    g = torch.Generator(device=DEV).manual_seed(C)
    kw.update(lidar_features=torch.randn(C, N, features, generator=g, device=DEV), **options)
    if C > 1:
        for k in ("viewmats", "raster_pts", "linear_velocity", "angular_velocity", "rolling_shutter_time"):
            kw[k] = kw[k].repeat(C, *([1] * (kw[k].dim() - 1)))
        kw["viewmats"][:, 0, 3] += torch.arange(C, device=DEV) * 1.0

    def wanted(images):
        every = _all_of(images)
        return every if at < 0 else [w if i == at else None for i, w in enumerate(every)]

    leaves = ("means", "quats", "scales", "opacities") + (("lidar_features",) if at in (-1, 0) else ())
    _twice(monkeypatch, "_native_lidar_frame", splatad_b200.lidar_rasterization, kw, leaves, wanted)
