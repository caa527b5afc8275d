"""Beta path factor kernel against the 160-digit references and the tensor form.

Tolerances: the golden test's (float32 rounds once: 6e-8, bounded by 3e-6; float64 2e-12). Against the tensor form in
float64 the factor goes through the same log-Gamma: 1e-13.
"""

import json
from pathlib import Path

import pytest
import torch

from r2splat_b200 import _beta, _fused

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_kernel_matches_160_digit_references(device, dtype):
    data = torch.tensor(json.loads((GOLDEN / "beta_references.json").read_text())["rows"], dtype=dtype, device=device)
    gamma = data[:, 0].contiguous()
    tol = 3e-6 if dtype == torch.float32 else 2e-12
    torch.testing.assert_close(_fused.beta_path_ratio(gamma), data[:, 1], atol=0, rtol=tol)
    torch.testing.assert_close(_fused.beta_path_log_grad(gamma), data[:, 2], atol=0, rtol=tol)


@pytest.mark.parametrize("n", [1, 255, 257, 10_000])
def test_kernel_matches_the_tensor_form(device, n):
    gamma = torch.logspace(-3, 4, n, dtype=torch.float64, device=device) if n > 1 else torch.full(
        (1,), 0.75, dtype=torch.float64, device=device)
    torch.testing.assert_close(_fused.beta_path_ratio(gamma), _beta.beta_path_ratio(gamma), atol=0, rtol=1e-13)
    # The tensor form subtracts two digamma values of size ln z: 4e-16 ln z / (1 / (2 z)), below 1e-12 at z = 33.
    torch.testing.assert_close(_fused.beta_path_log_grad(gamma), _beta.beta_path_log_grad(gamma), atol=0, rtol=1e-12)
    f32 = gamma.float()
    assert torch.equal(_fused.beta_path_ratio(f32), _beta.beta_path_ratio(f32))
