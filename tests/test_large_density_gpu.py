"""Variance VJPs of fp32 Gaussians whose squared density leaves the range of floats: the uncertainty adjoints are
density^2 times sums that may be zero or small, and stay finite.

Tolerance: the values are sums of products of one sign (the adjoint is positive), each factor rounded a few times, so
fp32 and float64 agree to far better than 1e-3 of each value; records at the contribution threshold aside, which weigh
nothing at these densities."""

import pytest
import torch

import r2splat_b200 as r2s
from r2splat_b200 import scenes

pytestmark = pytest.mark.gpu


def _uncertainty_gradient(device, operation, dtype, adjoint):
    n = 300
    means, quats, scales, dens, _, q = scenes.random_primitives(n, 13, 0.05, 0.2, uncertainty_max=0.1)
    dens = dens * 1e21
    args = [t.to(device=device, dtype=dtype) for t in (means, quats, scales, dens)]
    q = q.to(device=device, dtype=dtype)
    if operation == "rasterize":
        viewmats, Ks = (t.to(device=device, dtype=dtype) for t in scenes.orbit_cameras(2, 3.0, 90.0, 64, 64))
        out, ctx = r2s.rasterize_fwd(*args, viewmats, Ks, (64, 64), uncertainty=q, detach_variance=True)
        bwd = r2s.rasterize_bwd
    else:
        out, ctx = r2s.voxelize_fwd(*args, (32, 32, 32), volume_extent=(1.0, 1.0, 1.0), uncertainty=q,
                                    detach_variance=True)
        bwd = r2s.voxelize_bwd
    return bwd(ctx, None, torch.full_like(out[0], adjoint)).uncertainty


@pytest.mark.parametrize("operation", ["rasterize", "voxelize"])
def test_uncertainty_adjoints_stay_finite(device, operation):
    zero = _uncertainty_gradient(device, operation, torch.float32, 0.0)
    assert bool((zero == 0).all())
    small = _uncertainty_gradient(device, operation, torch.float32, 1e-20).double()
    truth = _uncertainty_gradient(device, operation, torch.float64, 1e-20)
    assert float(truth.max()) < 1e38 and float(truth.min()) >= 0
    torch.testing.assert_close(small, truth, rtol=1e-3, atol=0)
