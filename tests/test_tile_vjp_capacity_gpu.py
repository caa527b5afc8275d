"""r2s_raster_tile_bwd with the intersection count on the device: the gradients of the host-count form, bit for bit, where
the lists fit; zeros where they overflowed, whatever the slots hold."""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spare", [0, 500, -1])
def test_count_on_the_device(device, spare):
    n, c, h, w = 900, 3, 61, 85
    means, quats, scales, dens, _, q = (t.to(device) if t is not None else None for t in
                                        scenes.random_primitives(n, 21, 0.04, 0.3, uncertainty_max=0.1))
    viewmats, Ks = (t.to(device) for t in scenes.orbit_cameras(c, 3.0, 100.0, w, h))
    _, state = _fused.raster_forward(means, quats, scales, dens, viewmats, Ks, w, h, None, q, 1e-8, 3.0)
    gen = torch.Generator(device=device).manual_seed(4)
    v, vv = (torch.randn((c, h, w), device=device, generator=gen) for _ in range(2))
    m, stream = state.n_isects, torch.cuda.current_stream(device).cuda_stream
    ty, tx = state.offsets.shape[1:]

    def vjp(offsets, ids, count, n_used, capacity):
        slots = torch.full((capacity, 8), float("nan"), device=device)
        grads = torch.full((c, n, 8), float("nan"), device=device)
        unc = torch.full((c, n), float("nan"), device=device)
        _backend.call("r2s_raster_tile_bwd", _ptr(state.records), _ptr(state.extra["rects"]), _ptr(q), 0,
                      _ptr(offsets), _ptr(ids), count, n_used, _ptr(state.extra["cum"]), _ptr(v), _ptr(vv), c, n, w, h,
                      16, tx, ty, _ptr(slots), capacity, _ptr(grads), _ptr(unc), stream)
        return grads, unc

    capacity = m + spare
    n_used = torch.empty(1, dtype=torch.int64, device=device)
    overflow = torch.zeros(1, dtype=torch.int32, device=device)
    ids64 = torch.empty(capacity, dtype=torch.int64, device=device)
    ids = torch.empty(capacity, dtype=torch.int32, device=device)
    offsets = torch.empty_like(state.offsets)
    ws = _fused._ws(_backend.library().r2s_isect_emit_workspace(capacity, c * tx * ty), device)
    _backend.call("r2s_raster_emit_capacity", _ptr(state.extra["rects"]), c, n, tx, ty, _ptr(state.extra["cum"]),
                  capacity, _ptr(n_used), _ptr(overflow), _ptr(ids64), _ptr(ids), _ptr(offsets), _ptr(ws), ws.numel(),
                  stream)
    got = vjp(offsets, ids, capacity, _ptr(n_used), capacity)
    assert int(n_used) == (m if spare >= 0 else 0) and int(overflow) == int(spare < 0)
    if spare >= 0:
        for a, b in zip(got, vjp(state.offsets, state.flatten_ids, m, None, m)):
            assert torch.equal(a, b)
    else:
        assert bool((got[0] == 0).all()) and bool((got[1] == 0).all())
