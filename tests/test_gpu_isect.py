"""Bit-exact parity of tile intersection (tiles per Gaussian, sorted isect ids, flatten ids,
offsets) between the CUDA library and the CPU oracle / the reference's golden vectors."""

import math

import numpy as np
import pytest
import torch

from gpu_util import DEV, launched, n, t

pytestmark = pytest.mark.gpu


def _check(got, want, label):
    for name, a, b in zip(("tiles_per_gauss", "isect_ids", "flatten_ids", "isect_offsets"), got, want):
        a = n(a)
        assert a.shape == b.shape, f"{label} {name}: shape {a.shape} vs {b.shape}"
        if not np.array_equal(a, b):
            bad = np.nonzero(a.reshape(-1) != b.reshape(-1))[0]
            raise AssertionError(f"{label} {name}: {bad.size} of {a.size} entries differ, first at {bad[0]}: "
                                 f"got {a.reshape(-1)[bad[0]]} want {b.reshape(-1)[bad[0]]}")


def _run_cam(means2d, radii, depths, ts, tw, th, **kw):
    from splatad_b200 import ops
    C = kw.get("n_cameras") or means2d.shape[0]
    tpg, ids, flat = ops.isect_tiles(t(means2d), t(radii, torch.int32), t(depths), ts, tw, th, **kw)
    offs = ops.isect_offset_encode(ids, C, tw, th)
    # the offsets handed over by the fill equal the ones recomputed from the ids alone
    assert torch.equal(offs, ops.isect_offset_encode(ids.clone(), C, tw, th))
    return tpg, ids, flat, offs


def _run_lidar(means2d, radii, depths, eb, res, min_az, **kw):
    from splatad_b200 import ops
    C = kw.get("n_cameras") or means2d.shape[0]
    tpg, ids, flat = ops.isect_lidar_tiles(t(means2d), t(radii), t(depths), t(eb), res, min_az, **kw)
    n_az = math.ceil(360 / res)
    offs = ops.isect_offset_encode(ids, C, n_az, len(eb) - 1)
    assert torch.equal(offs, ops.isect_offset_encode(ids.clone(), C, n_az, len(eb) - 1))
    return tpg, ids, flat, offs


def test_isect_tiles_golden(golden):
    g = golden("isect_tiles")
    got = _run_cam(g["means2d"], g["radii"], g["depths"], int(g["tile_size"]), int(g["tile_width"]), int(g["tile_height"]))
    _check(got, [g[k] for k in ("tiles_per_gauss", "isect_ids", "flatten_ids", "isect_offsets")], "golden camera")


@pytest.mark.parametrize("name", ["isect_lidar_tiles", "isect_lidar_tiles_wrap"])
def test_isect_lidar_tiles_golden(golden, name):
    g = golden(name)
    got = _run_lidar(g["means2d"], g["radii"], g["depths"], g["elev_boundaries"], float(g["tile_azim_resolution"]),
                     float(g["min_azimuth"]))
    _check(got, [g[k] for k in ("tiles_per_gauss", "isect_ids", "flatten_ids", "isect_offsets")], name)


@pytest.mark.parametrize("C,N,W,H,ts", [(1, 1, 64, 64, 16), (2, 5000, 640, 480, 16), (3, 70000, 1920, 1080, 16),
                                         (1, 3000, 100, 60, 7), (1, 6000, 1100, 200, 16), (2, 9000, 300, 250, 16)])
def test_isect_tiles_vs_oracle(C, N, W, H, ts):
    from oracle import isect
    g = torch.Generator().manual_seed(C * 1000 + N)
    means2d = (torch.rand(C, N, 2, generator=g) * 1.4 - 0.2) * torch.tensor([W, H])
    radii = torch.randint(0, 60, (C, N, 2), generator=g, dtype=torch.int32)
    radii[:, ::9, 0] = 0
    depths = torch.rand(C, N, generator=g) * 50
    depths[:, 1::4] = depths[:, 0::4][:, : depths[:, 1::4].shape[1]]  # equal depths: ties keep flatten order
    tw, th = math.ceil(W / ts), math.ceil(H / ts)
    want = list(isect.isect_tiles(n(means2d), n(radii), n(depths), ts, tw, th))
    want.append(isect.isect_offset_encode(want[1], C, tw, th))
    got = _run_cam(means2d, radii, depths, ts, tw, th)
    _check(got, want, f"camera C={C} N={N}")
    # unsorted variant: emission in flatten order
    from splatad_b200 import ops
    tpg, ids, flat = ops.isect_tiles(t(means2d), t(radii, torch.int32), t(depths), ts, tw, th, sort=False)
    w = isect.isect_tiles(n(means2d), n(radii), n(depths), ts, tw, th, sort=False)
    _check((tpg, ids, flat), w, f"camera unsorted C={C} N={N}")


def test_isect_tiles_packed():
    from oracle import isect
    C, N, W, H, ts = 3, 20000, 640, 480, 16
    g = torch.Generator().manual_seed(77)
    nnz = 30000
    cam = torch.sort(torch.randint(0, C, (nnz,), generator=g)).values
    gau = torch.randint(0, N, (nnz,), generator=g)
    means2d = (torch.rand(nnz, 2, generator=g) * 1.2 - 0.1) * torch.tensor([W, H])
    radii = torch.randint(1, 40, (nnz, 2), generator=g, dtype=torch.int32)
    depths = torch.rand(nnz, generator=g) * 50
    tw, th = math.ceil(W / ts), math.ceil(H / ts)
    want = list(isect.isect_tiles(n(means2d), n(radii), n(depths), ts, tw, th, n_cameras=C, camera_ids=n(cam)))
    want.append(isect.isect_offset_encode(want[1], C, tw, th))
    got = _run_cam(means2d, radii, depths, ts, tw, th, packed=True, n_cameras=C, camera_ids=cam.to(DEV),
                   gaussian_ids=gau.to(DEV))
    _check(got, want, "camera packed")


@pytest.mark.parametrize("C,N", [(1, 1), (1, 4000), (2, 60000)])
def test_isect_lidar_tiles_vs_oracle(C, N):
    from oracle import isect
    from splatad_b200 import scenes
    g = torch.Generator().manual_seed(C * 100 + N)
    elev = scenes.beams_128()
    eb = scenes.elevation_boundaries(elev, 8)
    means2d = torch.stack([torch.rand(C, N, generator=g) * 360 - 180, torch.rand(C, N, generator=g) * 44 - 27], -1)
    radii = torch.rand(C, N, 2, generator=g) * torch.tensor([12.0, 4.0])
    radii[:, ::50, 0] = 200.0 + torch.rand(C, len(range(0, N, 50)), generator=g) * 300  # more than a full turn
    radii[:, ::11, 0] = 0
    depths = torch.rand(C, N, generator=g) * 80
    depths[:, 1::4] = depths[:, 0::4][:, : depths[:, 1::4].shape[1]]
    res = 0.2 * 32
    want = list(isect.isect_lidar_tiles(n(means2d), n(radii), n(depths), n(eb), res, -180.0))
    n_az = math.ceil(360 / res)
    want.append(isect.isect_offset_encode(want[1], C, n_az, len(eb) - 1))
    got = _run_lidar(means2d, radii, depths, eb, res, -180.0)
    _check(got, want, f"lidar C={C} N={N}")


def test_isect_empty_and_invisible():
    from splatad_b200 import ops
    z2 = torch.zeros(2, 0, 2, device=DEV)
    tpg, ids, flat = ops.isect_tiles(z2, z2.int(), torch.zeros(2, 0, device=DEV), 16, 4, 4)
    assert tpg.shape == (2, 0) and ids.numel() == 0 and flat.numel() == 0
    offs = ops.isect_offset_encode(ids, 2, 4, 4)
    assert offs.shape == (2, 4, 4) and int(offs.abs().sum()) == 0
    # all Gaussians culled
    m = torch.rand(1, 100, 2, device=DEV) * 64
    tpg, ids, flat = ops.isect_tiles(m, torch.zeros(1, 100, 2, dtype=torch.int32, device=DEV),
                                     torch.rand(1, 100, device=DEV), 16, 4, 4)
    assert int(tpg.sum()) == 0 and ids.numel() == 0


def test_isect_key_bits_error():
    from splatad_b200 import ops
    m = torch.rand(1, 10, 2, device=DEV)
    with pytest.raises(RuntimeError):
        ops.isect_tiles(m, torch.ones(1, 10, 2, dtype=torch.int32, device=DEV), torch.rand(1, 10, device=DEV),
                        1, 1 << 16, 1 << 16)


def test_two_deferred_intersections_outstanding():
    """Two deferred tile intersections alive at once - a camera call and a lidar call of different
    sizes, resolved in the opposite order: each reads ITS count (own pinned slot), so lengths, lists
    and offsets equal those of the two-step calls. A second pair runs on another stream, which has
    workspaces and capacity hints of its own."""
    from splatad_b200 import ops, scenes
    g = torch.Generator().manual_seed(5)
    C, N, W, H, ts = 2, 30_000, 640, 480, 16
    means2d = ((torch.rand(C, N, 2, generator=g) * 1.2 - 0.1) * torch.tensor([W, H])).to(DEV)
    radii = torch.randint(1, 40, (C, N, 2), generator=g, dtype=torch.int32).to(DEV)
    depths = (torch.rand(C, N, generator=g) * 50).to(DEV)
    tw, th = math.ceil(W / ts), math.ceil(H / ts)
    eb = scenes.elevation_boundaries(scenes.beams_128(), 8).to(DEV)
    M = 50_000
    l_means = torch.stack([torch.rand(1, M, generator=g) * 360 - 180, torch.rand(1, M, generator=g) * 44 - 27], -1).to(DEV)
    l_radii = (torch.rand(1, M, 2, generator=g) * torch.tensor([12.0, 4.0])).to(DEV)
    l_depths = (torch.rand(1, M, generator=g) * 80).to(DEV)
    res, n_az = 0.2 * 32, math.ceil(360 / (0.2 * 32))

    def cam():
        return ops.isect_tiles_deferred(means2d, radii, depths, ts, tw, th)

    def lid():
        return ops.isect_lidar_tiles_deferred(l_means, l_radii, l_depths, eb, res, -180.0)

    want_cam = ops.isect_tiles(means2d, radii, depths, ts, tw, th)
    want_lid = ops.isect_lidar_tiles(l_means, l_radii, l_depths, eb, res, -180.0)
    assert want_cam[1].numel() != want_lid[1].numel()

    def check_pair():
        cam().resolve(), lid().resolve()          # first frames of the two shapes: they leave the hints
        d_cam, d_lid = cam(), lid()               # both enqueued ahead of their counts, both outstanding
        assert d_cam._resolved is None and d_lid._resolved is None
        offs_lid, offs_cam = d_lid.offsets(16, n_az).clone(), d_cam.offsets(th, tw).clone()
        ids_l, flat_l = d_lid.resolve()           # opposite order
        ids_c, flat_c = d_cam.resolve()
        assert torch.equal(ids_c, want_cam[1]) and torch.equal(flat_c, want_cam[2])
        assert torch.equal(ids_l, want_lid[1]) and torch.equal(flat_l, want_lid[2])
        assert torch.equal(offs_cam, ops.isect_offset_encode(want_cam[1].clone(), C, tw, th))
        assert torch.equal(offs_lid, ops.isect_offset_encode(want_lid[1].clone(), 1, n_az, 16))
        assert torch.equal(d_cam.tiles_per_gauss, want_cam[0]) and torch.equal(d_lid.tiles_per_gauss, want_lid[0])

    check_pair()
    side = torch.cuda.Stream(DEV)
    side.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.stream(side):
        check_pair()
    side.synchronize()


@pytest.mark.parametrize("distinct", [1, 7, 150, 3000])
def test_depth_order_with_crowded_depths(distinct):
    """Depth order of the visible Gaussians when many depths coincide: with `distinct` different
    depths among 40,000 Gaussians a depth bucket holds from a dozen elements (ranked by counting) over
    a few hundred (bitonic network in shared memory) to thousands (beyond what the bucket sort
    orders: the plan says so and the lists come from the radix passes). All give the reference's
    order - ties by flatten index - bit for bit, for the two-step call, for a second, hinted frame of
    the same shape, and for the camera path."""
    from oracle import isect
    from splatad_b200 import ops, scenes
    C, N = 2, 20_000
    g = torch.Generator().manual_seed(100 + distinct)
    eb = scenes.elevation_boundaries(scenes.beams_128(), 8)
    means2d = torch.stack([torch.rand(C, N, generator=g) * 360 - 180, torch.rand(C, N, generator=g) * 44 - 27], -1)
    radii = torch.rand(C, N, 2, generator=g) * torch.tensor([9.0, 3.0])
    radii[:, ::13, 0] = 0
    levels = torch.rand(distinct, generator=g) * 80 + 0.5
    depths = levels[torch.randint(0, distinct, (C, N), generator=g)]
    res, n_az = 0.2 * 32, math.ceil(360 / (0.2 * 32))
    want = list(isect.isect_lidar_tiles(n(means2d), n(radii), n(depths), n(eb), res, -180.0))
    want.append(isect.isect_offset_encode(want[1], C, n_az, len(eb) - 1))
    ops._depth_sort_mode.clear()
    _check(_run_lidar(means2d, radii, depths, eb, res, -180.0), want, f"lidar, {distinct} depths")
    for _ in range(2):   # first deferred call leaves the hint, the second is enqueued ahead of its count
        d = ops.isect_lidar_tiles_deferred(t(means2d), t(radii), t(depths), t(eb), res, -180.0)
        got = d.resolve()
        if got is None:
            d = d.redo()
            got = d.resolve()
        _check((d.tiles_per_gauss, got[0], got[1]), want[:3], f"lidar deferred, {distinct} depths")
    crowded = 2 * N * 12 // 13 / distinct > 1024
    assert (2 in ops._depth_sort_mode.values()) == crowded
    # camera rectangles (one 640 x 480 camera: the row / column split; packed: three cameras)
    W, H, ts = 640, 480, 16
    m2 = (torch.rand(1, N, 2, generator=g) * 1.2 - 0.1) * torch.tensor([W, H])
    r2 = torch.randint(0, 40, (1, N, 2), generator=g, dtype=torch.int32)
    d2 = depths[:1]
    tw, th = math.ceil(W / ts), math.ceil(H / ts)
    want = list(isect.isect_tiles(n(m2), n(r2), n(d2), ts, tw, th))
    want.append(isect.isect_offset_encode(want[1], 1, tw, th))
    _check(_run_cam(m2, r2, d2, ts, tw, th), want, f"camera, {distinct} depths")


@pytest.mark.parametrize("lo,hi", [(0.0, 80.0), (10.0, 30.0), (0.0, 1.0e7), (79.0, 200.0)])
def test_depth_range_hint_never_changes_the_lists(lo, hi):
    """`splatad_isect_set_depth_range_hint` makes the depth buckets of the next plan span the given
    range instead of the measured one (and lets the rectangle count fill them): a range that fits, one
    that covers a slice of the depths, one far too wide and one that starts where the depths end all
    give the oracle's lists bit for bit - or, when an end bucket overflows, the status bit that sends
    the caller back to a plan without a hint."""
    import struct
    from oracle import isect
    from splatad_b200 import _lib, ops, scenes
    bits = lambda v: struct.unpack("<I", struct.pack("<f", v))[0]   # noqa: E731
    C, N = 1, 30_000
    g = torch.Generator().manual_seed(7)
    eb = scenes.elevation_boundaries(scenes.beams_128(), 8)
    means2d = torch.stack([torch.rand(C, N, generator=g) * 360 - 180, torch.rand(C, N, generator=g) * 44 - 27], -1)
    radii = torch.rand(C, N, 2, generator=g) * torch.tensor([9.0, 3.0])
    radii[:, ::7, 0] = 0
    depths = torch.rand(C, N, generator=g) * 80
    res, n_az = 0.2 * 32, math.ceil(360 / (0.2 * 32))
    want = list(isect.isect_lidar_tiles(n(means2d), n(radii), n(depths), n(eb), res, -180.0))
    want.append(isect.isect_offset_encode(want[1], C, n_az, len(eb) - 1))
    ops._depth_sort_mode.clear()
    _lib.load().splatad_isect_set_depth_range_hint(bits(lo), bits(hi))
    got = _run_lidar(means2d, radii, depths, eb, res, -180.0)   # an overflowing end bucket makes ops repeat the plan
    _check(got, want, f"lidar, depth range hint [{lo}, {hi}]")
    # a hint is consumed by one plan: the next call measures its own range again
    _check(_run_lidar(means2d, radii, depths, eb, res, -180.0), want, "lidar, after the hint")
    ops._depth_sort_mode.clear()   # an overflow above made this shape take the radix passes: not for other tests


@pytest.mark.parametrize("C,N,tw,th", [(1, 1, 1, 1), (1, 127, 3, 7), (1, 512, 4, 8), (2, 513, 5, 9), (3, 1500, 31, 17),
                                       (5, 300, 64, 40), (2, 1025, 1, 70), (130, 64, 9, 3)])
@pytest.mark.parametrize("packed", [False, True])
def test_block_split_at_the_edges_of_its_blocks(C, N, tw, th, packed):
    """The lists are built over blocks of 4 x 8 tiles, 512 entries per step-A block and 512 records per
    unit: grids one tile short of, at and beyond a block's edges, entry counts around the chunk sizes,
    sensors without a single entry, more sensors than a warp has lanes. Bit for bit the oracle's lists."""
    from oracle import isect
    from splatad_b200 import ops
    g = torch.Generator().manual_seed(C * 1000 + N)
    ts = 16
    m2 = (torch.rand(C, N, 2, generator=g) * 1.4 - 0.2) * torch.tensor([tw * ts, th * ts])
    r2 = torch.randint(0, 60, (C, N, 2), generator=g, dtype=torch.int32)
    r2[:, ::5] = r2[:, ::5] * 20                      # some cover the whole grid
    depths = torch.rand(C, N, generator=g) * 50 + 0.1
    depths[:, ::3] = depths[:, :1].clone()            # ties
    if C > 2:
        r2[1] = 0                                     # a sensor that sees nothing
    ops._depth_sort_mode.clear()
    if packed:
        keep = (r2[..., 0] > 0)
        cam = torch.nonzero(keep)[:, 0]
        args = (m2[keep], r2[keep], depths[keep])
        want = isect.isect_tiles(*(n(x) for x in args), ts, tw, th, n_cameras=C, camera_ids=n(cam))
        got = ops.isect_tiles(*(t(x) for x in args), ts, tw, th, packed=True, n_cameras=C, camera_ids=t(cam),
                              gaussian_ids=torch.zeros_like(t(cam)))
    else:
        want = isect.isect_tiles(n(m2), n(r2), n(depths), ts, tw, th)
        got = ops.isect_tiles(t(m2), t(r2), t(depths), ts, tw, th)
    for a, b, what in zip(got, want, ("tiles per Gaussian", "ids", "flatten ids")):
        assert np.array_equal(n(a), b), what
    offs = ops.isect_offset_encode(got[1], C, tw, th)
    assert np.array_equal(n(offs), isect.isect_offset_encode(want[1], C, tw, th))


@pytest.mark.parametrize("long_lists", [False, True])
@pytest.mark.parametrize("ids_off,flat_off", [(0, 0), (1, 0), (0, 1), (3, 2), (2, 4)])
@pytest.mark.parametrize("C,N,tw,th", [(1, 1, 1, 1), (1, 700, 4, 8), (2, 1400, 9, 9), (1, 3000, 13, 21), (2, 900, 70, 61)])
def test_lists_anywhere_in_memory(C, N, tw, th, ids_off, flat_off, long_lists, monkeypatch):
    """The list kernels write two entries at a time where both arrays are aligned for it, one otherwise; short and long runs of
    a tile, and room for so many entries that units of the longer kind are taken. Nothing outside the lists is written."""
    from splatad_b200 import _lib, ops
    g = torch.Generator().manual_seed(N + tw)
    W, H, ts = 16 * tw, 16 * th, 16
    means2d = torch.rand(C, N, 2, generator=g) * torch.tensor([W, H])
    radii = (torch.rand(C, N, 2, generator=g) ** 3 * 90).to(torch.int32) + 1
    depths = torch.rand(C, N, generator=g) * 30 + 0.5
    call, seen = ops._call, {}
    lists = dict(capacity=72_000_000 if long_lists else 1 << 18)
    ids = torch.full((lists["capacity"] + 16,), -7, dtype=torch.int64, device=DEV)
    flat = torch.full((lists["capacity"] + 16,), -7, dtype=torch.int32, device=DEV)
    starts = torch.full((C * tw * th + 16,), -7, dtype=torch.int32, device=DEV)
    fill_ws = torch.empty(_lib.load().splatad_isect_fill_workspace_bytes(lists["capacity"]), dtype=torch.uint8, device=DEV)

    def elsewhere(name, *args):
        if name == "splatad_isect_tiles_fill":
            *head, _, _, seen["n"], _, _, _, host, stream = args
            args = (*head, _lib.ptr(fill_ws), fill_ws.numel(), lists["capacity"], ids.data_ptr() + 8 * ids_off,
                    flat.data_ptr() + 4 * flat_off, starts.data_ptr() + 4 * flat_off, host, stream)
        return call(name, *args)

    want = _run_cam(means2d, radii, depths, ts, tw, th)
    monkeypatch.setattr(ops, "_call", elsewhere)
    ops.isect_tiles(t(means2d), t(radii), t(depths), ts, tw, th)
    n_isects = seen["n"]
    assert n_isects == want[1].numel() > 0
    assert torch.equal(ids[ids_off: ids_off + n_isects], want[1]) and torch.equal(flat[flat_off: flat_off + n_isects], want[2])
    n_tiles = C * tw * th
    assert torch.equal(starts[flat_off: flat_off + n_tiles], want[3].flatten()) and starts[flat_off + n_tiles] == n_isects
    for buffer, off, size in ((ids, ids_off, n_isects), (flat, flat_off, n_isects), (starts, flat_off, n_tiles + 1)):
        assert (buffer[:off] == -7).all() and (buffer[off + size: off + size + 8] == -7).all()


@pytest.mark.parametrize("ids_off,flat_off", [(0, 0), (1, 0), (2, 2), (2, 1)])
@pytest.mark.parametrize("capacity,kernel", [(11_000_000, "tile_scatter_kernel"), (11_100_000, "tile_scatter_kernel"),
                                             (41_900_000, "tile_scatter_kernel"), (42_000_000, "tile_scatter_kernel/1024")])
def test_list_kernels_by_the_room_for_entries(capacity, kernel, ids_off, flat_off, monkeypatch):
    """Plain stores, streaming stores, units of 1024 records: each side of the two lines, arrays aligned and not."""
    from splatad_b200 import _lib, ops
    C, N, tw, th = 2, 1400, 23, 17
    g = torch.Generator().manual_seed(3)
    means2d = torch.rand(C, N, 2, generator=g) * torch.tensor([16.0 * tw, 16.0 * th])
    radii = (torch.rand(C, N, 2, generator=g) ** 3 * 90).to(torch.int32) + 1
    depths = torch.rand(C, N, generator=g) * 30 + 0.5
    want = _run_cam(means2d, radii, depths, 16, tw, th)
    ids = torch.full((capacity + 8,), -7, dtype=torch.int64, device=DEV)
    flat = torch.full((capacity + 8,), -7, dtype=torch.int32, device=DEV)
    fill_ws = torch.empty(_lib.load().splatad_isect_fill_workspace_bytes(capacity), dtype=torch.uint8, device=DEV)
    call = ops._call

    def elsewhere(name, *args):
        if name == "splatad_isect_tiles_fill":
            *head, _, _, _, _, _, starts, host, stream = args
            args = (*head, _lib.ptr(fill_ws), fill_ws.numel(), capacity, ids.data_ptr() + 8 * ids_off, flat.data_ptr() + 4 * flat_off,
                    starts, host, stream)
        return call(name, *args)

    monkeypatch.setattr(ops, "_call", elsewhere)
    _, names = launched(lambda: ops.isect_tiles(t(means2d), t(radii), t(depths), 16, tw, th))
    assert kernel in names, names
    for buffer, off, lists in ((ids, ids_off, want[1]), (flat, flat_off, want[2])):
        size = lists.numel()
        assert torch.equal(buffer[off: off + size], lists)
        assert (buffer[:off] == -7).all() and (buffer[off + size: off + size + 8] == -7).all()


@pytest.mark.parametrize("radix", [False, True])
@pytest.mark.parametrize("C,N,tw,th,r", [(1, 5000, 60, 15, 200), (1, 300, 31, 30, 300), (1, 9000, 40, 30, 200), (2, 2600, 25, 18, 140), (3, 1500, 20, 15, 130),
                                         (6, 700, 30, 20, 300), (9, 600, 12, 9, 200), (20, 520, 9, 5, 250), (1, 5000, 20, 13, 90), (1, 5000, 60, 15, 9)])
def test_how_many_tiles_a_near_gaussian_covers(C, N, tw, th, r, radix, monkeypatch):
    """What a fill reports about the first entries in depth order is what their rectangles say."""
    from splatad_b200 import ops
    g = torch.Generator().manual_seed(C * N)
    means2d = (torch.rand(C, N, 2, generator=g) * 1.2 - 0.1) * torch.tensor([16.0 * tw, 16.0 * th])
    radii = torch.randint(0, 2 * r, (C, N, 2), generator=g, dtype=torch.int32)
    depths = torch.rand(C, N, generator=g) * 30 + 0.5
    args = (t(means2d), t(radii, torch.int32), t(depths), 16, tw, th)
    if radix:
        monkeypatch.setattr(ops, "_depth_sort_mode", _AlwaysRadix())
    tiles = n(ops.isect_tiles_deferred(*args).tiles_per_gauss).astype(np.int64)
    n_isects, listed, near = ops.isect_tiles_deferred(*args).flatten_ids._splatad_counts()
    if C * tw * th < 900 or r < 50:
        assert near == 0.0   # (few tiles, short lists: nobody asks)
        return
    assert n_isects == tiles.sum() and listed == (tiles > 0).sum()
    sensors, total, of = min(C, 8), 0, 0
    for i in range(sensors):
        c = i * (C // sensors)
        order = np.argsort(n(depths)[c], kind="stable")
        order, seen = order[tiles[c][order] > 0], 0
        for k in range({1: 8, 2: 4, 3: 2, 4: 2}.get(sensors, 1)):
            group = order[512 * k: 512 * (k + 1)]
            if seen >= 32 * tw * th:
                break
            seen, of = seen + tiles[c][group].sum(), of + len(group)
        total += seen
    assert near == pytest.approx(total / of, rel=1e-6)


def test_near_tiles_are_always_answered(monkeypatch):
    """Where no kernel reports them - lists that outgrow their room, a grid beyond the block split, unsorted output, lidar tiles, nothing to
    list - the answer is 0, and a request is never left for the next call. (Short lists alone go without an answer.)"""
    from splatad_b200 import _lib, ops, scenes
    lib = _lib.load()
    words = torch.zeros(1, dtype=torch.int64).pin_memory()
    monkeypatch.setattr(_lib, "NearRequest", lambda device: float)   # this test asks itself
    g = torch.Generator().manual_seed(4)

    def answered(sequence, call):
        words[0] = -1
        lib.splatad_isect_set_near_tiles(words.data_ptr(), sequence)
        call()
        torch.cuda.synchronize()
        assert int(words[0]) >> 32 == sequence, sequence
        return int(words[0]) & 0xFFFFFFFF

    def cam(N=900, tw=20, th=10, r=600, **kw):
        means2d = torch.rand(1, N, 2, generator=g) * torch.tensor([16.0 * tw, 16.0 * th])
        radii = torch.randint(1, r, (1, N, 2), generator=g, dtype=torch.int32)
        return ops.isect_tiles(t(means2d), t(radii, torch.int32), t(torch.rand(1, N, generator=g)), 16, tw, th, **kw)

    assert answered(1, cam) > 0
    assert answered(2, lambda: cam(sort=False)) == 0
    assert answered(3, lambda: cam(tw=256, th=136)) == 0
    eb = scenes.elevation_boundaries(scenes.beams_128(), 8)
    assert answered(4, lambda: _run_lidar(torch.rand(1, 500, 2, generator=g) * 20, torch.rand(1, 500, 2, generator=g) + 1, torch.rand(1, 500, generator=g),
                                          eb, 6.4, -180.0)) == 0
    call = ops._call

    def short(name, *args):   # room for three entries
        if name == "splatad_isect_tiles_fill":
            args = (*args[:-6], 3, *args[-5:])
        return call(name, *args)

    with monkeypatch.context() as patch:
        patch.setattr(ops, "_call", short)
        assert answered(5, cam) == 0
    p = _lib.ptr
    one = torch.zeros(8, device=DEV)
    assert answered(6, lambda: lib.splatad_isect_tiles_fill(1, 0, 0, *[p(one)] * 4, 16, 4, 4, 1, p(one), p(one), p(one), 32, 8, p(one), p(one), None, None,
                                                            None)) == 0
    words[0] = 0
    lib.splatad_isect_set_near_tiles(words.data_ptr(), 7)
    cam(r=30)
    cam()                                             # nothing is asked for any more
    torch.cuda.synchronize()
    assert int(words[0]) == 0


@pytest.mark.parametrize("turns", [0.3, 0.99, 1.0, 1.01, 2.4, 4.5])
def test_block_split_of_rectangles_around_the_turn(turns):
    """Lidar rectangles that wrap past the last azimuth tile, end just short of or just past a full
    turn, and go round more than once (their tiles then list the Gaussian once per turn)."""
    from oracle import isect
    from splatad_b200 import ops, scenes
    C, N = 2, 700
    g = torch.Generator().manual_seed(int(turns * 100))
    eb = scenes.elevation_boundaries(scenes.beams_128(), 8)
    means2d = torch.stack([torch.rand(C, N, generator=g) * 360 - 180, torch.rand(C, N, generator=g) * 44 - 27], -1)
    radii = torch.rand(C, N, 2, generator=g) * torch.tensor([3.0, 3.0]) + 1e-3
    radii[:, ::4, 0] = 180.0 * turns * (0.98 + 0.04 * torch.rand(C, radii[:, ::4].shape[1], generator=g))
    depths = torch.rand(C, N, generator=g) * 50 + 0.1
    res, n_az = 0.2 * 32, math.ceil(360 / (0.2 * 32))
    want = list(isect.isect_lidar_tiles(n(means2d), n(radii), n(depths), n(eb), res, -180.0))
    want.append(isect.isect_offset_encode(want[1], C, n_az, len(eb) - 1))
    ops._depth_sort_mode.clear()
    _check(_run_lidar(means2d, radii, depths, eb, res, -180.0), want, f"{turns} turns")


class _AlwaysRadix(dict):
    """Every shape is taken for one whose depths are too crowded for the buckets."""

    def get(self, key, default=None):
        return 2


@pytest.mark.parametrize("C,N,tw,th", [(1, 1, 1, 1), (1, 513, 3, 7), (2, 513, 5, 9), (3, 1500, 31, 17), (256, 40, 3, 9),
                                       (257, 40, 9, 3), (600, 9, 2, 2)])
@pytest.mark.parametrize("packed", [False, True])
def test_crowded_depths_take_the_block_split(C, N, tw, th, packed, monkeypatch):
    """Behind the radix passes the entries are grouped by sensor - by none, one or two further passes - and split
    as behind the buckets. Bit for bit the oracle's lists, by the same kernels."""
    import ctypes
    from oracle import isect
    from splatad_b200 import _lib, ops
    g = torch.Generator().manual_seed(C * 1000 + N)
    ts = 16
    m2 = (torch.rand(C, N, 2, generator=g) * 1.4 - 0.2) * torch.tensor([tw * ts, th * ts])
    r2 = torch.randint(0, 60, (C, N, 2), generator=g, dtype=torch.int32)
    depths = torch.rand(C, N, generator=g) * 50 + 0.1
    depths[:, ::3] = depths[:, :1].clone()            # ties
    if C > 2:
        r2[1] = 0                                     # a sensor that sees nothing
    monkeypatch.setattr(ops, "_depth_sort_mode", _AlwaysRadix())
    lib = _lib.load()
    keep = r2[..., 0] > 0
    cam = torch.nonzero(keep)[:, 0]
    lib.splatad_profile_enable(1)
    try:
        if packed:
            want = isect.isect_tiles(n(m2[keep]), n(r2[keep]), n(depths[keep]), ts, tw, th, n_cameras=C, camera_ids=n(cam))
            got = ops.isect_tiles(t(m2[keep]), t(r2[keep], torch.int32), t(depths[keep]), ts, tw, th, packed=True, n_cameras=C,
                                  camera_ids=cam.to(DEV), gaussian_ids=torch.zeros_like(cam).to(DEV))
        else:
            want = isect.isect_tiles(n(m2), n(r2), n(depths), ts, tw, th)
            got = ops.isect_tiles(t(m2), t(r2, torch.int32), t(depths), ts, tw, th)
        torch.cuda.synchronize()
        report = ctypes.create_string_buffer(1 << 16)
        lib.splatad_profile_report(report, len(report))
    finally:
        lib.splatad_profile_enable(0)
    for a, b, what in zip(got, want, ("tiles per Gaussian", "ids", "flatten ids")):
        assert np.array_equal(n(a), b), what
    offs = ops.isect_offset_encode(got[1], C, tw, th)
    assert np.array_equal(n(offs), isect.isect_offset_encode(want[1], C, tw, th))
    names = report.value.decode()
    assert "depthsort_upsweep" in names and "tilesort_upsweep" not in names
    assert ("tile_scatter_kernel" in names) == (got[1].numel() > 0)
