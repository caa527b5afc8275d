"""Tile-parallel raster VJP (r2s_raster_tile_bwd) against the record walk of the same records in float64.

Well-conditioned records: a sample's relative error is below 4e-6 (exponent up to 17 at 6e-8, the fast exponential),
and a record of at most 4096 samples sums to below 4096 x 6e-8 = 2.5e-4 of its terms in the worst case, about 64 x
6e-8 x a few in the mean; entries that cancel are judged against the component's rms over all records: 1e-4 of |truth|
+ rms. Elongated records' exponents and position sums cancel by their condition number in any fp32 evaluation: there
the error may be as large as 1.5 times that of the fp32 record walk, which takes the same decisions.
"""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu

TOLERANCE = 1e-4


def _scene(device, n, cameras, height, width, scale, elongated=False):
    means, quats, scales, densities, _, _ = scenes.random_primitives(n, 5, scale, 0.4)
    if elongated:  # projected condition numbers past 1000: boxes of the whole tile, the strict walk
        scales[::2, 0] *= 60.0
        scales[::2, 1:] *= 0.3
    densities[::7] = 0.0
    viewmats, Ks = scenes.orbit_cameras(cameras, 3.0, 1.2 * max(height, width), width, height)
    return [t.to(device) for t in (means, quats, scales, densities, viewmats, Ks)]


def _record_walk(state, q, v, vv, detach, dtype):
    c, n = state.records.shape[:2]
    records, q, v, vv = (t.to(dtype) for t in (state.records, q, v, vv))
    grads = torch.empty((c, n, 8), dtype=dtype, device=v.device)
    unc = torch.empty((c, n), dtype=dtype, device=v.device)
    _backend.call("r2s_raster_record_bwd", int(dtype == torch.float64), _ptr(records), _ptr(state.extra["rects"]),
                  _ptr(q), 0, int(detach), _ptr(v), _ptr(vv), c, n, state.width, state.height, state.tile_size,
                  _ptr(grads), None, _ptr(unc), torch.cuda.current_stream().cuda_stream)
    return grads, unc


def _tile_walk(state, q, v, vv, detach):
    c, n = state.records.shape[:2]
    grads = torch.full((c, n, 8), float("nan"), device=state.records.device)
    unc = torch.full((c, n), float("nan"), device=grads.device)
    m = state.n_isects
    slots = torch.full((max(m, 1), 8), float("nan"), device=grads.device)
    _backend.call("r2s_raster_tile_bwd", _ptr(state.records), _ptr(state.extra["rects"]), _ptr(q), int(detach),
                  _ptr(state.offsets), _ptr(state.flatten_ids), m, None, _ptr(state.extra["cum"]), _ptr(v), _ptr(vv),
                  c, n, state.width, state.height, state.tile_size, state.offsets.shape[2], state.offsets.shape[1],
                  _ptr(slots), slots.shape[0], _ptr(grads), _ptr(unc), torch.cuda.current_stream().cuda_stream)
    return grads, unc


def _error(x, truth):
    """Largest error of each component, against |truth| + rms."""
    dims = (0, 1)
    rms = truth.square().mean(dim=dims).sqrt()
    return ((x.double() - truth).abs() / (truth.abs() + rms).clamp_min(1e-300)).amax(dim=dims)


def _check(state, q, v, vv, detach, v_zero=None):
    """The tile walk's result, checked; ``v_zero`` stands for a null image adjoint in the record walk."""
    mine = _tile_walk(state, q, v, vv, detach)
    truth = _record_walk(state, q, v if v_zero is None else v_zero, vv, detach, torch.float64)
    other = _record_walk(state, q, v if v_zero is None else v_zero, vv, detach, torch.float32)
    for x, t, o in zip(mine, truth, other):
        x, t, o = (y[..., :7] if y.dim() == 3 else y for y in (x, t, o))
        assert torch.isfinite(x).all()
        assert (_error(x, t) <= (1.5 * _error(o, t)).clamp_min(TOLERANCE)).all()
    return mine


@pytest.mark.parametrize("variance", ["attached", "detached"])
@pytest.mark.parametrize("n,cameras,height,width,tile,scale,elongated", [
    (1, 1, 1, 1, 8, 0.3, False),            # one pixel
    (33, 2, 37, 53, 8, 0.05, False),        # tiles of one block, ragged edges
    (33, 3, 37, 53, 32, 0.05, False),       # 16 blocks a tile
    (2000, 1, 40, 40, 16, 0.15, False),     # lists of hundreds: several batches a warp, shared by CTAs
    (700, 3, 130, 71, 16, 0.02, True),      # boxes of whole tiles
    (500, 2, 64, 64, 16, 0.003, False),     # sub-pixel records, tiles without any
])
def test_tile_vjp_matches_the_record_walk(device, n, cameras, height, width, tile, scale, elongated, variance):
    means, quats, scales, densities, viewmats, Ks = _scene(device, n, cameras, height, width, scale, elongated)
    gen = torch.Generator().manual_seed(9)
    q = (0.1 * torch.rand((n,), generator=gen)).to(device)
    _, state = _fused.raster_forward(means, quats, scales, densities, viewmats, Ks, width, height, None, q, 1e-8, 3.0,
                                     tile)
    v = torch.randn((cameras, height, width), generator=gen).to(device)
    vv = (0.1 * torch.randn((cameras, height, width), generator=gen)).to(device)
    mine, _ = _check(state, q, v, vv, variance == "detached")
    again, _ = _tile_walk(state, q, v, vv, variance == "detached")
    assert torch.equal(mine, again)


def test_no_intersections_and_null_image_adjoint(device):
    means, quats, scales, densities, viewmats, Ks = _scene(device, 40, 2, 48, 48, 0.02)
    q = torch.full((40,), 0.05, device=device)
    behind = viewmats.clone()
    behind[:, 2, 3] -= 10.0  # every primitive behind its camera
    vv = torch.ones((2, 48, 48), device=device)
    for views, empty in ((behind, True), (viewmats, False)):
        _, state = _fused.raster_forward(means, quats, scales, densities, views, Ks, 48, 48, None, q, 1e-8, 3.0)
        assert (state.n_isects == 0) == empty
        _check(state, q, None, vv, False, v_zero=torch.zeros((2, 48, 48), device=device))
