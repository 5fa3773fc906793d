"""Frames through the native host side (``csrc/host/frames.cpp``): from the second frame of a shape on, one call
enqueues the frame and puts its own two nodes into the autograd graph. Whatever it takes, its images, lists,
gradients and refusals are those of the individual ops."""

import pytest
import torch

from gpu_util import DEV

pytestmark = pytest.mark.gpu


def _to_gpu(cfg):
    return {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in cfg.items()}


def _forget():
    """No frame has a predecessor: the next one is rendered by the individual ops."""
    from splatad_b200 import ops
    for hint in (ops._isect_count_hint, ops._packed_nnz_hint, ops._depth_range_hint, ops._depth_sort_mode):
        hint.clear()


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
