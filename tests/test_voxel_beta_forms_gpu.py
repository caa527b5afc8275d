"""The fp32 Beta voxel kernels in each of their forms: slabs of a tile in the forward, shares of a list in the VJP, packed
and gathered records, slots and atomics. The general kernels, which the first tile layers of a grid take when rendered
alone (their lists are a prefix of the whole grid's), give the expected values.

Forward and slots: the same operations in the same order, so bit for bit. Atomics: the slots of a primitive in any order,
so off by at most (slots - 1) x 2^-24 of the sum of their magnitudes; twice that is allowed, for the sum compared with."""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu

# shape, layers rendered alone, primitives, scale, pairs a tile (from, to), more than 16 tiles a primitive.
# Tiles 972 (four slabs), 2964 (two), 7650 (one).
CASES = [
    ((96, 65, 71), 4, 20_000, 0.03, 128, 1000, False),    # four shares
    ((96, 65, 71), 4, 1_500, 0.03, 1, 128, True),         # short lists
    ((150, 95, 101), 2, 60_000, 0.03, 128, 1000, True),   # four shares
    ((150, 95, 101), 2, 20_000, 0.015, 32, 128, False),   # two
    ((150, 95, 101), 2, 4_000, 0.01, 0, 32, False),       # one
    ((150, 95, 101), 2, 1_200, 0.12, 16, 128, True),      # large records
    ((200, 130, 140), 1, 60_000, 0.025, 64, 1000, True),  # two shares
    ((200, 130, 140), 1, 3_000, 0.025, 0, 64, True),      # one
]


@pytest.mark.parametrize("variance", [False, True])
@pytest.mark.parametrize("shape,layers,n,scale,least,most,large", CASES)
def test_forms_equal_the_general_kernels(device, shape, layers, n, scale, least, most, large, variance):
    means, quats, scales, dens, b, q = scenes.random_primitives(n, 17, scale, 0.4, beta_range=(0.5, 4.0),
                                                                uncertainty_max=0.1)
    scales[::7, 0] *= 8.0  # needles of every bound
    scales[1:9, 0] *= 100.0
    scales[9:13, :2] *= 60.0  # sheets
    dens[::11] = 0.0
    means, quats, scales, dens, b, q = (t.to(device) for t in (means, quats, scales, dens, b, q))
    extent, center = torch.ones(3, device=device), torch.zeros(3, device=device)
    covars = _fused._covariances(quats, scales)
    records, offsets, _, flatten_ids, m, means_v, radii, cum = _fused.voxel_intersections(
        means, covars, dens, b, q if variance else None, extent, center, shape, 1e-8, 1.0, 8)
    records[3::17, 4] *= -1.0  # indefinite conics
    records[6::29, 3] *= -1.0
    tx, ty, tz = _fused._voxel_tiles(shape, 8)
    assert tx * ty * layers <= 444 and least * tx * ty * tz <= m < most * tx * ty * tz and (m > 16 * n) == large
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
            _backend.call("r2s_voxel_render_bwd_slots", 0, _ptr(records), 1, 0, _ptr(offsets), _ptr(flatten_ids),
                          count, None, _ptr(means_v), _ptr(radii), _ptr(cum), _ptr(v), _ptr(vv), n, *grid,
                          _ptr(slots), m, _ptr(grads), stream)
        return vol, var, slots, grads

    gathered, staged = run(shape[0], m, False), run(shape[0], m, True)
    part_m = int(offsets.flatten()[tx * ty * layers])
    part = run(8 * layers, part_m, True)
    for a, c, rows in zip(gathered[:2], staged[:2], part[:2]):
        if a is not None:
            assert torch.equal(a, c) and torch.equal(a[:8 * layers], rows)
            assert float(a.abs().max()) > 0 and not bool((a == -7.0).any())
    columns = 12 if variance else 11
    assert not bool(staged[2].isnan().any())  # every pair's slot is written
    assert torch.equal(gathered[2][:, :columns], staged[2][:, :columns])
    assert torch.equal(gathered[3], staged[3])
    first = ~part[2][:, 0].isnan()  # the slots of the first layers' pairs
    assert int(first.sum()) == part_m > 0
    assert torch.equal(staged[2][first][:, :columns], part[2][first][:, :columns])

    # The low-level form adds the same partial sums with atomics.
    atomics = torch.zeros((n, 16), device=device)
    _backend.call("r2s_voxel_render_bwd", 0, _ptr(records), 1, 0, _ptr(offsets), _ptr(flatten_ids), _ptr(v), _ptr(vv), n,
                  m, shape[2], shape[1], shape[0], 8, tx, ty, tz, _ptr(atomics), stream)
    magnitude = torch.cat((torch.zeros((1, 12), dtype=torch.float64, device=device),
                           staged[2].double().abs().cumsum(0)))
    last, begin = cum, torch.cat((cum.new_zeros(1), cum[:-1]))
    bound = 2.0**-23 * (last - begin).double()[:, None] * (magnitude[last] - magnitude[begin])
    error = (atomics[:, :columns].double() - staged[3][:, :columns].double()).abs()
    # The cumulative sums of magnitudes round too: 2^-40 of their total covers it.
    assert bool((error <= bound[:, :columns] + 2.0**-40 * magnitude[-1, :columns]).all())
