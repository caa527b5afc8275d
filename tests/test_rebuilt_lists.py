"""The variance VJP of fp32 Gaussians where the forward's tile lists are no longer held: they are built again from the
rectangles at hand and those rectangles' own count, never from a count kept from the forward.

The same records in the same lists give the same sums in the same order, so every comparison is bit for bit."""

import pytest
import torch

import r2splat_b200 as r2s
from r2splat_b200 import _fused, explicit, scenes
from r2splat_b200 import autograd as ag
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

FIELDS = ("means", "quats", "scales", "densities", "uncertainty")
SIZE = (90, 117)


def test_the_lists_are_sized_by_the_rectangles_own_count(monkeypatch):
    """On the CPU: a state whose recorded count is stale. The buffers handed to the emission have the fresh count."""
    rects = torch.tensor([[[0, 0, 2, 3], [1, 1, 1, 1], [3, 2, 8, 3]], [[0, 0, 0, 0], [5, 5, 6, 7], [0, 0, 8, 6]]],
                         dtype=torch.int16)
    counts = [6, 0, 5, 0, 2, 48]
    emitted = {}

    def call(name, *args):
        assert name == "r2s_raster_emit"
        emitted.update(n=args[6], cum=args[5])

    monkeypatch.setattr(_fused, "_stream", lambda device: 0)
    monkeypatch.setattr(_fused._backend, "call", call)
    monkeypatch.setattr(_fused._backend, "library", lambda: type("L", (), {
        "r2s_isect_emit_workspace": staticmethod(lambda m, keys: m)})())
    monkeypatch.setattr(_fused, "_raster_scan", lambda c: c.flatten().to(torch.int64).cumsum(0))
    monkeypatch.setattr(_fused, "_read_total", lambda cum: int(cum[-1]))
    monkeypatch.setattr(torch.cuda.nvtx, "range_push", lambda name: None)
    monkeypatch.setattr(torch.cuda.nvtx, "range_pop", lambda: None)
    for stale in (None, 3, 10_000):
        state = _fused.RasterState(None, None, None, None, None, None, stale, 117, 90, 16, extra={"rects": rects})
        ids, offsets, cum, slots = _fused._raster_vjp_lists(state, torch.float32, False, True)
        assert emitted["n"] == ids.numel() == slots.shape[0] == sum(counts)
        assert cum.tolist() == torch.tensor(counts).cumsum(0).tolist()
        assert offsets.shape == (2, 6, 8)


def _scene(device, n=3000, cameras=5):
    means, quats, scales, dens, _, q = scenes.random_primitives(n, 7, 0.04, 0.4, uncertainty_max=0.1)
    viewmats, Ks = scenes.orbit_cameras(cameras, 3.0, 130.0, SIZE[1], SIZE[0])
    gen = torch.Generator().manual_seed(3)
    v, vv = (torch.randn((cameras,) + SIZE, generator=gen) for _ in range(2))
    return [t.to(device) for t in (means, quats, scales, dens, q, viewmats, Ks, v, 0.1 * vv)]


def _explicit(device, viewmats=None, release=False):
    means, quats, scales, dens, q, views, Ks, v, vv = _scene(device)
    _, ctx = r2s.rasterize_fwd(means, quats, scales, dens, views if viewmats is None else viewmats, Ks, SIZE,
                               uncertainty=q)
    if release:
        explicit.release_intersection_lists(ctx)
    g = r2s.rasterize_bwd(ctx, v, vv)
    return [getattr(g, f) for f in FIELDS]


def _graph(device, recompute):
    means, quats, scales, dens, q, views, Ks, v, vv = _scene(device)
    leaves = [t.requires_grad_() for t in (means, quats, scales, dens, q)]
    image, variance = ag.rasterize(*leaves[:4], views, Ks, SIZE, uncertainty=leaves[4], recompute=recompute)
    return leaves, views, (image * v).sum() + (variance * vv).sum()


@pytest.mark.gpu
def test_released_recomputed_and_second_backwards_equal_the_kept_lists(device):
    kept = _explicit(device)
    assert all(float(g.abs().max()) > 0 for g in kept)
    leaves, _, loss = _graph(device, True)
    recomputed = torch.autograd.grad(loss, leaves)
    leaves, _, loss = _graph(device, False)
    first = torch.autograd.grad(loss, leaves, retain_graph=True)
    second = torch.autograd.grad(loss, leaves)
    for other in (_explicit(device, release=True), recomputed, first, second):
        for a, b in zip(kept, other):
            assert torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("distance", [1.4, 6.0, -10.0])  # more intersections than in the forward, fewer, none
@pytest.mark.parametrize("second", [False, True])
def test_cameras_written_since_the_forward(device, distance, second):
    leaves, views, loss = _graph(device, not second)
    if second:
        torch.autograd.grad(loss, leaves, retain_graph=True)
    views[:, 2, 3] = distance
    grads = torch.autograd.grad(loss, leaves)
    for a, b in zip(grads, _explicit(device, viewmats=views.clone())):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_saved_tensors_stored_in_16_bits(device):
    """A hook that narrows what the graph keeps: the backward's rectangles differ from the forward's."""
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().to(torch.bfloat16), lambda t: t.float()):
        leaves, views, loss = _graph(device, True)
    grads = torch.autograd.grad(loss, leaves)
    _, _, _, _, _, _, Ks, v, vv = _scene(device)
    _, ctx = r2s.rasterize_fwd(*(t.detach().to(torch.bfloat16).float() for t in leaves[:4]), views, Ks, SIZE,
                               uncertainty=leaves[4].detach().to(torch.bfloat16).float())
    g = r2s.rasterize_bwd(ctx, v.to(torch.bfloat16).float(), vv.to(torch.bfloat16).float())
    for a, name in zip(grads, FIELDS):
        assert torch.equal(a, getattr(g, name))


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [2, 3])
def test_emission_writes_nothing_past_its_count(device, dims):
    """A count below the scan's last entry: keys, ids and lists stay inside what that count sizes."""
    means, quats, scales, dens, q, views, Ks, _, _ = _scene(device)
    covars = _fused._covariances(quats, scales)
    stream = _fused._stream(device)
    if dims == 2:
        _, rects, counts = _fused._raster_project(means, covars, dens, None, None, views, Ks, SIZE[1], SIZE[0], 1e-8,
                                                  3.0, 16)
        cum, keys = _fused._raster_scan(counts), 5 * 6 * 8
    else:
        extent, center = torch.ones(3, device=device), torch.zeros(3, device=device)
        _, means_v, radii, _, cum = _fused._voxel_project(means, covars, dens, None, None, extent, center,
                                                          (40, 48, 56), 1e-8, 3.0, 8)
        keys = 5 * 6 * 7
    total = int(cum[-1])
    m, guard = total // 2, total  # the guard holds what a write by the scan would reach
    nbytes = int(_backend.library().r2s_isect_emit_workspace(m, keys))
    ws = torch.full((nbytes + 16 * total,), 7, dtype=torch.uint8, device=device)
    ids = torch.full((m + guard,), -3, dtype=torch.int64, device=device)
    flat = torch.full((m + guard,), -3, dtype=torch.int32, device=device)
    offsets = torch.empty((keys,), dtype=torch.int32, device=device)
    if dims == 2:
        _backend.call("r2s_raster_emit", _ptr(rects), 5, means.shape[0], 8, 6, _ptr(cum), m, _ptr(ids), _ptr(flat),
                      _ptr(offsets), _ptr(ws), nbytes, stream)
    else:
        _backend.call("r2s_isect_tiles_3d_emit", 0, _ptr(means_v), _ptr(radii), means.shape[0], 8, 7, 6, 5, _ptr(cum),
                      m, _ptr(ids), _ptr(flat), _ptr(offsets), _ptr(ws), nbytes, stream)
    assert bool((ids[m:] == -3).all()) and bool((flat[m:] == -3).all())
    assert bool((ws[nbytes:] == 7).all())
    assert bool((flat[:m] >= 0).all()) and int(offsets.max()) <= m


@pytest.mark.gpu
def test_the_scan_is_kept_only_for_the_vjp_that_reads_it(device):
    means, quats, scales, dens, q, views, Ks, _, _ = _scene(device)
    beta = torch.full_like(dens, 1.5)
    for dtype, options, kept in ((torch.float32, {"uncertainty": q}, True), (torch.float32, {}, False),
                                 (torch.float32, {"uncertainty": q, "beta": beta}, False),
                                 (torch.float64, {"uncertainty": q}, False)):
        args = [t.to(dtype) for t in (means, quats, scales, dens, views, Ks)]
        _, ctx = r2s.rasterize_fwd(*args, SIZE, **{k: t.to(dtype) for k, t in options.items()})
        state = ctx.buffers["state"]
        assert ("cum" in state.extra) == kept
        explicit.release_intersection_lists(ctx)
        assert "cum" not in state.extra


@pytest.mark.gpu
@pytest.mark.parametrize("release", [False, True])
def test_without_room_for_slots_or_lists_the_records_are_walked(device, monkeypatch, release):
    """Over the slot budget, or with an allocation refused: the record walk's gradients, bit for bit the same in
    either case, and the tile walk's to rounding (5e-5 in the relative 2-norm: see the tile walk's own test)."""
    tiles = _explicit(device, release=release)

    def no_room(*args):
        raise torch.OutOfMemoryError("no room")

    with monkeypatch.context() as patch:
        patch.setattr(_fused, "RASTER_SLOT_BUDGET_BYTES", 32)
        walked = _explicit(device, release=release)
    for name in ("_raster_slots", "_raster_lists") if release else ("_raster_slots",):
        with monkeypatch.context() as patch:
            means, quats, scales, dens, q, views, Ks, v, vv = _scene(device)
            _, ctx = r2s.rasterize_fwd(means, quats, scales, dens, views, Ks, SIZE, uncertainty=q)
            if release:
                explicit.release_intersection_lists(ctx)
            patch.setattr(_fused, name, no_room)
            g = r2s.rasterize_bwd(ctx, v, vv)
        for a, b in zip(walked, (getattr(g, f) for f in FIELDS)):
            assert torch.equal(a, b)
    for a, b in zip(walked, tiles):
        assert float((a - b).norm()) <= 5e-5 * float(a.norm())


def test_rule_for_the_tile_walk():
    def takes(isects, records, lists, visible=None):
        asked = []

        def count():
            asked.append(True)
            return visible

        taken = _fused.raster_vjp_takes_tiles(isects, records, lists, count)
        assert bool(asked) == (visible is not None)  # counted only where it can change the answer
        return taken

    assert takes(0, 0, 10**6)  # nothing to walk
    assert takes(9, 4, 4096) and not takes(8, 4, 4096)  # 2.25 tiles a record
    assert not takes(65_536, 65_536, 100)
    assert takes(225_000, 200_000, 100, visible=100_000) and not takes(225_000, 200_000, 100, visible=100_001)
    # 65,536 lists of 3.7 tiles a record: 18 records a list pay for the lists, nine do not.
    for records, pays in ((18, True), (9, False)):
        n = 65536 * records
        assert takes(n, n * 10 // 37, 65536, visible=None if pays else n * 10 // 37) == pays
        assert takes(n, n, 65536, visible=n * 10 // 37) == pays
    budget = _fused.RASTER_SLOT_BUDGET_BYTES // _fused.RASTER_SLOT_BYTES
    assert takes(budget, 1000, 1) and not takes(budget + 1, 1000, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [0, 1, 255, 2049, 3_000_001])
def test_records_with_tiles_are_counted(device, n):
    rects = torch.randint(0, 3, (n, 4), generator=torch.Generator().manual_seed(n)).to(device, torch.int16)
    x0, y0, x1, y1 = rects.unbind(-1)
    assert _fused._read_visible(rects) == int(((x1 > x0) & (y1 > y0)).sum())


@pytest.mark.gpu
def test_partly_visible_scene_counts_and_takes_tiles(device, monkeypatch):
    """More than 65,536 records, most of them off the detectors: fewer than 2.25 tiles a record, more a visible one."""
    n, size = 30_000, (24, 640)
    means, quats, scales, dens, _, q = (None if t is None else t.to(device) for t in
                                        scenes.random_primitives(n, 9, 0.02, 0.3, uncertainty_max=0.1))
    viewmats, Ks = (t.to(device) for t in scenes.orbit_cameras(3, 3.0, 700.0, size[1], size[0]))
    v = torch.randn((3,) + size, device=device, generator=torch.Generator(device=device).manual_seed(1))
    decisions, rule = [], _fused.raster_vjp_takes_tiles

    def watched(isects, records, lists, count):
        decisions.append((isects, records, rule(isects, records, lists, count)))
        return decisions[-1][2]

    monkeypatch.setattr(_fused, "raster_vjp_takes_tiles", watched)
    grads = []
    for release in (False, True):
        _, ctx = r2s.rasterize_fwd(means, quats, scales, dens, viewmats, Ks, size, uncertainty=q)
        if release:
            explicit.release_intersection_lists(ctx)
        grads.append(r2s.rasterize_bwd(ctx, v, v))
    assert len(decisions) == 2 and all(4 * m < 9 * c and c > 65_536 and taken for m, c, taken in decisions)
    for name in FIELDS:
        assert torch.equal(getattr(grads[0], name), getattr(grads[1], name))


@pytest.mark.gpu
def test_small_footprints_take_the_record_walk(device, monkeypatch):
    """Records of about one tile each: the gradients of the record walk, bit for bit, kept, released or recomputed."""
    original = _scene

    def small(device, n=3000, cameras=5):
        scene = original(device, n, cameras)
        scene[2] = scene[2] * 0.02
        return scene

    monkeypatch.setitem(globals(), "_scene", small)
    kept = _explicit(device)
    leaves, _, loss = _graph(device, True)
    others = [_explicit(device, release=True), torch.autograd.grad(loss, leaves)]
    monkeypatch.setattr(_fused, "raster_vjp_takes_tiles", lambda *args: False)
    others.append(_explicit(device))
    monkeypatch.setattr(_fused, "raster_vjp_takes_tiles", lambda *args: True)
    tiles = _explicit(device)
    for other in others:
        for a, b in zip(kept, other):
            assert torch.equal(a, b)
    assert not all(torch.equal(a, b) for a, b in zip(kept, tiles))
