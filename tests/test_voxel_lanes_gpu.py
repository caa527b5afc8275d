"""The fp32 Gaussian voxel VJP with one lane per (tile, primitive) pair, with the variance branch, against float64.

Tolerance. A sample's exponent is a sum of six products, each factor and sum rounded once (at most 12 roundings of 2^-24
relative to the terms), and the terms exceed their sum by at most the conic's condition number: below 40 in these scenes
(axis ratios up to about 6), over exponents of at most 14 ln-units. That is 12 * 2^-24 * 14 * 40 = 4e-4 for a worst
sample; rounding errors of the sums' terms are independent, and a norm over thousands of gradient entries of hundreds of
samples each averages them by well over a factor of 10. Samples at the threshold (1e-6) weigh nothing. So 5e-5 in the
relative 2-norm."""

import pytest
import torch

import r2splat_b200 as r2s
from r2splat_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("detach", [False, True])
@pytest.mark.parametrize("image_adjoint", [False, True])
@pytest.mark.parametrize("shape,n", [((8, 8, 8), 1), ((9, 7, 15), 33), ((40, 33, 26), 4000), ((16, 16, 24), 1000)])
def test_variance_vjp_matches_float64(device, shape, n, image_adjoint, detach):
    prims = list(scenes.random_primitives(n, 11, 0.05, 0.35, uncertainty_max=0.2))
    means, quats, scales, dens, _, q = prims
    dens[3::10] = 0.0
    gen = torch.Generator().manual_seed(2)
    v, vv = (torch.randn(shape, generator=gen) for _ in range(2))

    def grads(dtype):
        args = [t.to(device=device, dtype=dtype) for t in (means, quats, scales, dens)]
        _, ctx = r2s.voxelize_fwd(*args, shape, volume_extent=(1.0, 1.0, 1.0),
                                  uncertainty=q.to(device=device, dtype=dtype), detach_variance=detach)
        return r2s.voxelize_bwd(ctx, v.to(device=device, dtype=dtype) if image_adjoint else None,
                                vv.to(device=device, dtype=dtype))

    ours, ref = grads(torch.float32), grads(torch.float64)
    for name in ("means", "quats", "scales", "densities", "uncertainty"):
        a, b = getattr(ours, name).double(), getattr(ref, name)
        if not image_adjoint and detach and name != "uncertainty":
            assert float(a.abs().max()) == 0.0 and float(b.abs().max()) == 0.0
            continue
        assert float((a - b).norm()) <= 5e-5 * float(b.norm()), name
        assert float(b.norm()) > 0
