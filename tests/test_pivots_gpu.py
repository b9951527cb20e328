"""FAST, batched and mixed factors on matrices that are hard on them -- nearly collinear
neighbouring columns, values near the ends of the exponent range, rows whose entries differ
by orders of magnitude -- against the entrywise bound of a column-by-column factor."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def _collinear(n, start, gap, seed):
    """Correlation matrix of n features: feature start + 1 is feature start plus gap times
    another direction, the others correlate with both."""
    rng = np.random.default_rng([n, start, seed])
    F = rng.standard_normal((8 * n + 64, n))
    z = rng.standard_normal(len(F))
    F[:, start + 1] = F[:, start] + gap * z
    for j in range(n):
        if j not in (start, start + 1):
            F[:, j] = 0.3 * F[:, j] + rng.standard_normal() * F[:, start] + rng.standard_normal() * z
    F /= np.sqrt((F * F).sum(0))
    a = (F.T @ F).astype(np.float32)
    return np.tril(a) + np.tril(a, -1).T


def _factor(gpu_lla, path, a):
    torch = _torch()
    n = len(a)
    if path == "batch":
        plan = gpu_lla.BatchPlan(np.array([n], np.int32), np.array([1], np.int32), "f32" if a.dtype == np.float32 else "f64")
        ap, bp = plan.pack([a], [np.ones((n, 1), a.dtype)])
        A, B = torch.from_numpy(ap.copy()).cuda(), torch.from_numpy(bp.copy()).cuda()
        info = torch.empty(1, dtype=torch.int32, device="cuda")
        plan.solve(A, B, info)
        torch.cuda.synchronize()
        return A.cpu().numpy()[:n * n].reshape((n, n), order="F"), int(info.item())
    L = torch.from_numpy(a.copy()).cuda().T
    if path == "device":
        info = gpu_lla.potrf_device(L, algo=gpu_lla.ALGO_FAST)
    else:
        info = gpu_lla.spotrf_mixed_device(L, update="bf16x6")
    torch.cuda.synchronize()
    return L.cpu().numpy(), int(info.item())


@pytest.mark.parametrize("path", ["device", "batch", "mixed"])
@pytest.mark.parametrize("n,gap", [(4, 1e-2), (4, 3e-3), (8, 1e-2), (8, 3e-3), (16, 1e-2), (32, 1e-2), (64, 1e-2)])
@pytest.mark.parametrize("start", [0, 1, "last"])
def test_collinear_neighbours(gpu_lla, path, n, gap, start):
    """|L L^T - A|_ij over sqrt(a_ii a_jj): quotients and scalings by approximate reciprocals cost
    at most 8 eps a product, the sums (worst case n eps / 2) n eps / 8 as they add up in earnest."""
    start = n - 4 if start == "last" else start
    for seed in range(3):
        a = _collinear(n, start, gap, seed)
        fac, info = _factor(gpu_lla, path, a)
        assert info == -1
        low = np.tril(fac).astype(np.float64)
        scale = np.sqrt(np.diag(a).astype(np.float64))
        err = np.abs(low @ low.T - a) / scale[:, None] / scale[None, :]
        assert err.max() <= (8 + n / 8) * np.finfo(np.float32).eps, (seed, err.max())


@pytest.mark.parametrize("path", ["device", "batch"])
@pytest.mark.parametrize("n", [1, 2, 5, 33, 65, 200])
@pytest.mark.parametrize("scale", [2.0**126, 1.9 * 2.0**126, 2.0**-100])
def test_pivots_near_the_ends_of_the_range(gpu_lla, path, n, scale):
    """Pivots above 2^126, whose reciprocals are subnormal, and tiny ones: the same bound."""
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, 2 * n))
    g /= np.sqrt((g * g).sum(1))[:, None]
    a = (g @ g.T * scale).astype(np.float32)
    a = np.tril(a) + np.tril(a, -1).T
    fac, info = _factor(gpu_lla, path, a)
    assert info == -1
    low = np.tril(fac).astype(np.float64)
    err = np.abs(low @ low.T - a) / scale
    assert err.max() <= (8 + n / 8) * np.finfo(np.float32).eps, err.max()


@pytest.mark.parametrize("path,n", [("device", 65), ("device", 192), ("device", 500), ("batch", 33), ("batch", 200), ("batch", 256)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("groups", [2, 5])
def test_weakly_coupled_interleaved_groups(gpu_lla, path, n, dtype, groups):
    """Rows large in the columns of their own group and small in the others', which alternate, under a
    diagonal scaling over six orders: the digits of a row hold its entries to a fraction of the
    row's largest, so the bound is against sqrt(a_ii a_jj), as it is for FMAs, and no entry's own
    relative accuracy is promised."""
    rng = np.random.default_rng(n + groups)
    g = rng.standard_normal((n, 2 * n))
    own = (np.arange(n) % groups)[:, None] == (np.arange(2 * n) % groups)[None, :]
    g = np.where(own, g, g * (1e-6 if dtype == np.float64 else 1e-3))
    g /= np.sqrt((g * g).sum(1))[:, None]
    d = 10.0 ** rng.uniform(-3, 3, n)
    a = ((g @ g.T) * d[:, None] * d[None, :]).astype(dtype)
    a = np.tril(a) + np.tril(a, -1).T
    fac, info = _factor(gpu_lla, path, a)
    assert info == -1
    low = np.tril(fac).astype(np.longdouble)
    scale = np.sqrt(np.diag(a).astype(np.float64))
    err = np.abs((low @ low.T - a).astype(np.float64)) / scale[:, None] / scale[None, :]
    assert err.max() <= (8 + n / 8) * np.finfo(dtype).eps, err.max()
