"""Device paths at the sizes where they can go wrong (edges of tiles,
remainders, both sides of a dispatch rule), against FP64 references."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def _spd(torch, n, shift, seed):
    """G G^T / n + shift I (kappa about 4 / shift), FP64, symmetric."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    G = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = G @ G.T / n
    A = (A + A.T) * 0.5
    A.diagonal().add_(shift)
    return A, g


@pytest.mark.parametrize("n,m", [(65, 1), (600, 3), (1000, 64), (1500, 70)])
@pytest.mark.parametrize("shift", [1.0, 0.01])
def test_refined_slices_of_well_conditioned_systems_converge(gpu_lla, n, m, shift):
    """One correction takes a well-conditioned system to its target: the exact-slice
    residual has to resolve that error (no stall, no fallback to plain FP64)."""
    torch = _torch()
    A, g = _spd(torch, n, shift, n + m)
    B = torch.randn(m, n, dtype=torch.float64, device="cuda", generator=g).T
    X = torch.empty(m, n, dtype=torch.float64, device="cuda").T
    rep = gpu_lla.posv_refined_device(A.T, B, X, residual="slices")
    torch.cuda.synchronize()
    assert rep["converged"] == 1 and rep["fell_back"] == 0 and rep["iterations"] <= 3, rep
    R = B - A @ X
    be = (R.abs().amax(0) / (A.abs().sum(1).amax() * X.abs().amax(0) + B.abs().amax(0))).max()
    assert float(be) <= 1.1e-13  # the default tolerance, plus the check's own rounding
