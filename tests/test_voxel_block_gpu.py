"""The fp32 Gaussian voxel forward with a 4 x 2 x 2 block per lane (8^3 tiles, more than 592 of them) against the row form
that small grids take. Each sample's expression and rounding are the same in both, so the volumes agree bit for bit: the
lists of a grid's first tile layers are a prefix of the whole grid's, and on those alone the row form runs."""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu


def _render(records, offsets, flatten_ids, n, m, shape, variance, packed=None):
    depth, height, width = shape
    tx, ty, tz = _fused._voxel_tiles(shape, 8)
    volume = torch.full(shape, -7.0, device=records.device)
    var = torch.full(shape, -7.0, device=records.device) if variance else None
    stream = torch.cuda.current_stream(records.device).cuda_stream
    if packed is None:
        _backend.call("r2s_voxel_render", 0, _ptr(records), 0, _ptr(offsets), _ptr(flatten_ids), n, m, width, height,
                      depth, 8, tx, ty, tz, _ptr(volume), _ptr(var), stream)
    else:
        _backend.call("r2s_voxel_render_packed", 0, _ptr(packed), 0, _ptr(offsets), m, None, width, height, depth, 8, tx,
                      ty, tz, _ptr(volume), _ptr(var), stream)
    return volume, var


@pytest.mark.parametrize("variance", [False, True])
@pytest.mark.parametrize("shape,layers", [((96, 65, 71), 6), ((83, 72, 90), 5), ((600, 8, 65), 60)])
def test_block_form_equals_row_form_bitwise(device, shape, layers, variance):
    n = 12_000
    means, quats, scales, dens, _, q = scenes.random_primitives(n, 7, 0.02, 0.4, uncertainty_max=0.1)
    scales[::5, 0] *= 12.0  # elongated: the conic is not bounded
    dens[::11] = 0.0
    dens[5::13] = 5e-7  # never reaches the threshold
    means, quats, scales, dens, q = (t.to(device) for t in (means, quats, scales, dens, q))
    extent, center = torch.ones(3, device=device), torch.zeros(3, device=device)
    covars = _fused._covariances(quats, scales)
    records, offsets, _, flatten_ids, m, _, radii, cum = _fused.voxel_intersections(
        means, covars, dens, None, q if variance else None, extent, center, shape, 1e-8, 3.0, 8)
    # Entries the lists do not depend on: indefinite conics, entries whose products underflow or overflow, negative and
    # non-finite opacities. Columns: x, y, z, o, c00, c01, c02, c11, c12, c22.
    records[3::17, 4] *= -1.0
    records[4::19, 5:7] = 1e-25
    records[5::23, 9] = 3e30
    records[6::29, 3] *= -1.0
    records[7::4001, 3] = float("inf")
    records[8::4001, 7] = float("nan")
    tx, ty, tz = _fused._voxel_tiles(shape, 8)
    assert tx * ty * tz > 592 and tx * ty * layers <= 592
    assert int((offsets.flatten()[1:] - offsets.flatten()[:-1]).max()) > 96  # the stages are used again
    packed = _fused.pack_tile_records(records, offsets, flatten_ids, radii, cum, m, shape, 8)
    gathered = _render(records, offsets, flatten_ids, n, m, shape, variance)
    bulk = _render(records, offsets, flatten_ids, n, m, shape, variance, packed)
    m_part = int(offsets.flatten()[tx * ty * layers])
    part = _render(records, offsets, flatten_ids, n, m_part, (8 * layers,) + shape[1:], variance)
    for whole, staged, rows in zip(gathered, bulk, part):
        if whole is None:
            continue
        assert torch.equal(whole.view(torch.int32), staged.view(torch.int32))
        assert torch.equal(torch.nan_to_num(whole[:8 * layers], nan=3.0), torch.nan_to_num(rows, nan=3.0))
        assert torch.equal(whole[:8 * layers].isnan(), rows.isnan())
        assert float(whole.nan_to_num().abs().max()) > 0 and not bool((whole == -7.0).any())
