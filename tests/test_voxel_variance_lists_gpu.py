"""The fp32 Gaussian voxel VJP with the variance branch on both sides of the list length at which it changes kernel (4,000
pairs and ten a tile), against float64: the tolerance of the lane form's own test, 5e-5 in the relative 2-norm, whose
derivation (rounded exponents of conics with condition numbers below 40) does not depend on the kernel."""

import pytest
import torch

import r2splat_b200 as r2s
from r2splat_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,short", [(120, True), (900, False)])
@pytest.mark.parametrize("shape", [(40, 37, 40), (17, 160, 24)])
def test_variance_vjp_either_side(device, shape, n, short):
    means, quats, scales, dens, _, q = scenes.random_primitives(n, 6, 0.04, 0.35, uncertainty_max=0.2)
    gen = torch.Generator().manual_seed(8)
    v, vv = (torch.randn(shape, generator=gen) for _ in range(2))
    tiles = 1
    for size in shape:
        tiles *= (size + 7) // 8

    def grads(dtype):
        args = [t.to(device=device, dtype=dtype) for t in (means, quats, scales, dens)]
        _, ctx = r2s.voxelize_fwd(*args, shape, volume_extent=(1.0, 1.0, 1.0), uncertainty=q.to(device, dtype))
        assert (ctx.buffers["state"].n_isects < 4000 + 10 * tiles) == short
        return r2s.voxelize_bwd(ctx, v.to(device, dtype), vv.to(device, dtype))

    ours, ref = grads(torch.float32), grads(torch.float64)
    for name in ("means", "quats", "scales", "densities", "uncertainty"):
        a, b = getattr(ours, name).double(), getattr(ref, name)
        assert float((a - b).norm()) <= 5e-5 * float(b.norm()) and float(b.norm()) > 0, name
