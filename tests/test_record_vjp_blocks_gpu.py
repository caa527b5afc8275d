"""The record VJP's split over blocks: many records give each block several runs of records, few give it one. A record's
sums do not depend on the records that share its warp, so a launch over all cameras and launches over a few cameras each
(other runs per block, other neighbours, other mixes of bounded and elongated conics in a warp) agree bit for bit."""

import pytest
import torch

import r2splat_b200 as r2s
from r2splat_b200 import scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta,variance", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("views", [1, 14, 96])  # 36,001, 0.5 and 3.5 million records
def test_record_vjp_is_independent_of_the_split(device, views, beta, variance):
    n, h, w = 36_001, 40, 56
    means, quats, scales, dens, b, q = scenes.random_primitives(
        n, 3, 0.02, 0.4, beta_range=(0.5, 4.0) if beta else None, uncertainty_max=0.1 if variance else None)
    scales[::7, 0] *= 60.0  # conics that are not bounded, among those that are
    means, quats, scales, dens, b, q = (None if t is None else t.to(device) for t in (means, quats, scales, dens, b, q))
    viewmats, Ks = (t.to(device) for t in scenes.orbit_cameras(views, 3.0, 120.0, w, h))
    _, ctx = r2s.rasterize_fwd(means, quats, scales, dens, viewmats, Ks, (h, w), beta=b, uncertainty=q)
    state = ctx.buffers["state"]
    rects, records = state.extra["rects"], state.records
    gen = torch.Generator(device=device).manual_seed(1)
    v = torch.randn((views, h, w), generator=gen, device=device)
    vv = torch.randn((views, h, w), generator=gen, device=device) if variance else None

    def run(step):
        grads = torch.full((views, n, 8), float("nan"), device=device)
        unc = torch.full((views, n), float("nan"), device=device) if variance else None
        for a in range(0, views, step):
            e = min(a + step, views)
            _backend.call("r2s_raster_record_bwd", 0, _ptr(records[a:e]), _ptr(rects[a:e]), _ptr(q), int(beta), 0,
                          _ptr(v[a:e]), _ptr(vv[a:e]) if variance else None, e - a, n, w, h, state.tile_size,
                          _ptr(grads[a:e]), None, _ptr(unc[a:e]) if variance else None,
                          torch.cuda.current_stream(device).cuda_stream)
        return grads, unc

    whole, parts = run(views), run(5 if views > 5 else 1)
    for x, y in zip(whole, parts):
        if x is not None:
            assert not bool(x.isnan().any()) and torch.equal(x, y)
    assert float(whole[0].abs().max()) > 0
