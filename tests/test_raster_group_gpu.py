"""Group-of-lanes raster forward (tile sizes 8, 16, 32 in fp32) against the float64 kernel on the same records and lists.

A well-conditioned sample's alpha is off by at most 12 x 6e-8 (exponent) + 1e-6 (fast exponential or power) relative,
a pixel sums up to a few hundred positive terms: 2e-5 of its value. A sample on the other side of the 1e-5 threshold in
float64 moves a pixel by 1e-5; four such are allowed. Records with condition numbers of thousands (the strict walk) are
off by that number x 6e-8 x the exponent: 1e-2 of the value, and only show whether a record is missing or misplaced.
"""

import pytest
import torch

from r2splat_b200 import _fused, scenes
from r2splat_b200._fused import _ptr
from r2splat_b200.cuda import _backend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta,variance", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("n,cameras,height,width,tile,batch,scale,strict", [
    (1, 1, 1, 1, 8, 256, 0.3, False),
    (300, 2, 37, 53, 8, 256, 0.05, False),      # one warp a tile, ragged edges
    (300, 3, 37, 53, 16, 5, 0.05, False),       # batches of 8 records: list padding, many batches
    (1500, 1, 40, 72, 16, 256, 0.2, False),     # lists of several full batches
    (700, 33, 130, 71, 32, 256, 0.05, False),   # 495 lists: the pair kernel still
    (700, 35, 130, 71, 32, 256, 0.05, False),   # 525 lists: 8x8 blocks
    (400, 3, 66, 50, 16, 256, 0.02, True),      # elongated records: whole tiles, strict walk
])
def test_group_forward_matches_float64(device, n, cameras, height, width, tile, batch, scale, strict, beta, variance):
    means, quats, scales, densities, b, q = scenes.random_primitives(
        n, 3, scale, 0.4, beta_range=(0.5, 4.0) if beta else None, uncertainty_max=0.1 if variance else None)
    if strict:
        scales[::2, 0] *= 60.0
        scales[::2, 1:] *= 0.5
    densities[::5] = 0.0
    viewmats, Ks = scenes.orbit_cameras(cameras, 3.0, 1.2 * max(height, width), width, height)
    to = (lambda t: None if t is None else t.to(device))
    means, quats, scales, densities, b, q, viewmats, Ks = map(to, (means, quats, scales, densities, b, q, viewmats, Ks))
    _, state = _fused.raster_forward(means, quats, scales, densities, viewmats, Ks, width, height, b, q, 1e-8,
                                     1.0 if beta else 3.0, tile)
    n_used = torch.tensor([state.n_isects], dtype=torch.int64, device=device)

    def render(dtype):
        image = torch.empty((cameras, height, width), dtype=dtype, device=device)
        var = torch.empty_like(image) if variance else None
        records, unc = state.records.to(dtype), None if q is None else q.to(dtype)
        _backend.call("r2s_raster_render_capacity", int(dtype == torch.float64), _ptr(records), _ptr(unc), int(beta),
                      _ptr(state.offsets), _ptr(state.flatten_ids), _ptr(n_used), cameras, n, width, height, tile,
                      state.offsets.shape[2], state.offsets.shape[1], batch, _ptr(image), _ptr(var),
                      torch.cuda.current_stream().cuda_stream)
        return [x for x in (image, var) if x is not None]

    relative = 1e-2 if strict else 2e-5
    for mine, truth in zip(render(torch.float32), render(torch.float64)):
        assert ((mine.double() - truth).abs() <= relative * truth.abs() + 4e-5).all()
