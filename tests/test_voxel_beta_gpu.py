"""The fp32 Beta voxel kernels that walk boxes (8^3 tiles, more than 444 of them) against the forms that small grids take.

Forward: each sample's expression and rounding are the same and a voxel adds its samples in list order. VJP: each slot's
sums are formed with the same rounding in the same order. So both agree bit for bit; a grid's first tile layers alone take
the general forms, and their lists are a prefix of the whole grid's."""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variance", [False, True])
@pytest.mark.parametrize("shape,layers", [((96, 65, 71), 4), ((83, 72, 90), 3), ((600, 8, 65), 48)])
def test_box_walks_equal_the_general_forms(device, shape, layers, variance):
    n = 20_000
    means, quats, scales, dens, b, q = scenes.random_primitives(n, 7, 0.03, 0.4, beta_range=(0.5, 4.0),
                                                                uncertainty_max=0.1)
    scales[::5, 0] *= 15.0  # needles: conics of the wider bound
    scales[2::50, 0] *= 200.0  # and of none
    dens[::11] = 0.0
    means, quats, scales, dens, b, q = (t.to(device) for t in (means, quats, scales, dens, b, q))
    extent, center = torch.ones(3, device=device), torch.zeros(3, device=device)
    covars = _fused._covariances(quats, scales)
    records, offsets, _, flatten_ids, m, means_v, radii, cum = _fused.voxel_intersections(
        means, covars, dens, b, q if variance else None, extent, center, shape, 1e-8, 1.0, 8)
    records[3::17, 4] *= -1.0  # indefinite conics
    records[6::29, 3] *= -1.0
    tx, ty, tz = _fused._voxel_tiles(shape, 8)
    assert tx * ty * tz > 444 >= tx * ty * layers
    packed = _fused.pack_tile_records(records, offsets, flatten_ids, radii, cum, m, shape, 8)
    stream = torch.cuda.current_stream(device).cuda_stream
    gen = torch.Generator(device=device).manual_seed(5)
    v = torch.randn(shape, generator=gen, device=device)
    vv = torch.randn(shape, generator=gen, device=device) if variance else None

    def run(depth, count, staged):
        dims = (depth,) + tuple(shape[1:])
        grid = (dims[2], dims[1], depth, 8, tx, ty, (depth + 7) // 8)
        vol = torch.full(dims, -7.0, device=device)
        var = torch.full(dims, -7.0, device=device) if variance else None
        slots = torch.full((m, 12), float("nan"), device=device)
        grads = torch.empty((n, 16), device=device)
        if staged:
            _backend.call("r2s_voxel_render_packed", 0, _ptr(packed), 1, _ptr(offsets), count, None, *grid, _ptr(vol),
                          _ptr(var), stream)
            _backend.call("r2s_voxel_render_bwd_packed", 0, _ptr(packed), 1, 0, _ptr(offsets), count, None, _ptr(cum),
                          _ptr(v), _ptr(vv), n, *grid, _ptr(slots), m, _ptr(grads), stream)
        else:
            _backend.call("r2s_voxel_render", 0, _ptr(records), 1, _ptr(offsets), _ptr(flatten_ids), n, count, *grid,
                          _ptr(vol), _ptr(var), stream)
            _backend.call("r2s_voxel_render_bwd_packed", 0, _ptr(packed), 1, 0, _ptr(offsets), count, None, _ptr(cum),
                          _ptr(v), _ptr(vv), n, *grid, _ptr(slots), m, _ptr(grads), stream)
        return vol, var, slots

    whole, staged = run(shape[0], m, False), run(shape[0], m, True)
    part_m = int(offsets.flatten()[tx * ty * layers])
    part = run(8 * layers, part_m, True)
    for a, c, rows in zip(whole[:2], staged[:2], part[:2]):
        if a is not None:
            assert torch.equal(a, c) and torch.equal(a[:8 * layers], rows)
            assert float(a.abs().max()) > 0 and not bool((a == -7.0).any())
    assert not bool(staged[2].isnan().any())  # every pair's slot is written
    first = ~part[2][:, 0].isnan()  # the slots of the first layers' pairs
    assert int(first.sum()) == part_m
    columns = 12 if variance else 11
    assert torch.equal(staged[2][first][:, :columns], part[2][first][:, :columns])
