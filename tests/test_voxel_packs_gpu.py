"""Which explicit voxel calls copy their records into list order, and that both forms give the same bits."""

import pytest
import torch

import r2splat_b200 as r2s
from r2splat_b200 import _fused, scenes

pytestmark = pytest.mark.gpu


def test_the_rule_lies_where_the_budgets_say():
    edge = _fused.VOXEL_GAUSSIAN_PACK_BYTES // 112  # 28 values of 4 bytes an intersection
    assert _fused.voxel_packs(torch.float32, False, 8, edge) and not _fused.voxel_packs(torch.float32, False, 8, edge + 1)
    large = _fused.VOXEL_PACK_BUDGET_BYTES // 112
    for dtype, beta, tile, most in ((torch.float32, True, 8, large), (torch.float32, False, 4, large),
                                    (torch.float64, False, 8, large // 2)):
        assert _fused.voxel_packs(dtype, beta, tile, most) and not _fused.voxel_packs(dtype, beta, tile, most + 1)


@pytest.mark.parametrize("variance", [False, True])
def test_gathered_gaussians_equal_packed_ones(device, monkeypatch, variance):
    means, quats, scales, dens, _, q = (None if t is None else t.to(device) for t in scenes.random_primitives(
        6000, 4, 0.03, 0.4, uncertainty_max=0.1 if variance else None))
    shape = (70, 77, 81)  # 990 tiles, ragged
    gen = torch.Generator(device=device).manual_seed(1)
    v, vv = (torch.randn(shape, generator=gen, device=device) for _ in range(2))
    results = []
    for budget in (1 << 40, 0):
        monkeypatch.setattr(_fused, "VOXEL_GAUSSIAN_PACK_BYTES", budget)
        out, ctx = r2s.voxelize_fwd(means, quats, scales, dens, shape, volume_extent=(1, 1, 1), uncertainty=q)
        assert (ctx.buffers["state"].packed is None) == (budget == 0)
        grads = r2s.voxelize_bwd(ctx, v, vv if variance else None)
        results.append([*(out if variance else (out,)), grads.means, grads.quats, grads.scales, grads.densities,
                        *([grads.uncertainty] if variance else [])])
    assert all(torch.equal(a, b) for a, b in zip(*results))
